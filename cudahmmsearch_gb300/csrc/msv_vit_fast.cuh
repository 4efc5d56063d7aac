// msv_vit_fast.cuh -- p7_ViterbiFilter with two nodes per register and fused
// add-and-maximum instructions, for profiles whose scores cannot wrap.
//
// The general kernels (msv_vit.cu) saturate every sum. Here every state value
// is kept at or above a floor F that no result can depend on, and the host
// checks from the profile's costs (VitFastPlan::build) that no 16-bit sum of a
// stored value and a cost can then leave the range downwards. A candidate and
// its maximum are one __viaddmax_s16x2, for two nodes at once:
//   M(k) = max(xB + BM(k), M'(k-1) + MM(k), I'(k-1) + IM(k), D'(k-1) + DM(k)) + e(k, x)
//   I(k) = max(M'(k) + MI(k), I'(k) + II(k), F)
//   D(k) = max(M(k-1) + MD(k-1), F), closed under D->D where the bound asks for it
// 9 instructions per two nodes instead of about 25 per node.
//
// Why the floor changes nothing. xB >= G = base + move(L) in every row (N's
// loop is 0), so a match cell's candidates are at least G + min BM = F; a
// predecessor below F, raised to F, still offers at most F (costs are <= 0),
// and I and D reach a score through a match cell only. M itself is stored
// exactly. Why nothing wraps upwards: before the emission no candidate
// exceeds the largest score so far; from the row where that score plus the
// largest emission could pass 32767, and on residues with emissions too low
// for a plain add (gap and other non-residue codes), the row runs its
// saturating variant. Padding nodes (past M, up to 64 W) have costs that keep
// them at or below the best real match cell of every row. The D->D closure is
// run whenever the largest D passes the profile's bound; running it more often
// changes no match cell, because the host checks that the bound covers every
// D->D->M step.
//
// Bound: the fused add-maximum runs at half rate (64 lanes per clock and SM);
// six per word of two nodes. The transition costs stay in registers across
// rows (up to 16 words per lane; wider models read them from shared memory),
// a row reads only its residue's emissions.
#pragma once
#include <cuda_runtime.h>

#include "msv_device.cuh"

namespace msvgb {

// Transition tables: BM MM IM DM (into the node), MD MI II (out of it), DD (into it).
constexpr int kFT = 8;
// Words per lane with the transitions in registers; above, in shared memory.
constexpr int kVitFastRegW = 16;

struct VitFastDev {
  int base_w, ddbound_w, xwE_move, xwE_loop, xwC_loop;
  int bm_min;               // smallest entry cost of a real node: F = base + move + bm_min
  int hot;                  // 32767 - twice the largest emission: no row can pass 32767 within the next two
  uint32_t low_res;         // residues whose emissions need the saturating row
  const uint32_t *trans;    // [kFT] rows of the lane layout below
  const uint32_t *emit;     // [NRES] rows
  const int16_t *move;      // [Lmax + 1]
};

// One row of W words per lane, lane-contiguous in 16-byte quads [q][32][4],
// then a pair [32][2] and a single [32] for the remainder: W * 32 words.
// Word w of lane l holds nodes l * 2W + w + 1 (low half) and l * 2W + W + w + 1.
__host__ __device__ constexpr int vitf_at(int W, int lane, int w) {
  return w < W / 4 * 4 ? (w / 4 * 32 + lane) * 4 + w % 4
       : (W % 4 >= 2 && w < W / 4 * 4 + 2) ? W / 4 * 128 + lane * 2 + (w - W / 4 * 4)
                                           : W / 4 * 128 + (W % 4 >= 2 ? 64 : 0) + lane;
}

// Words 4q .. 4q+3 of a row (the last call of a row takes the remainder).
template <int W>
__device__ __forceinline__ void vitf_load(uint32_t (&e)[W], const uint32_t *__restrict__ row, int lane, int q) {
  if (q < W / 4) {
    const uint4 v = *reinterpret_cast<const uint4 *>(row + (q * 32 + lane) * 4);
    e[4 * q] = v.x; e[4 * q + 1] = v.y; e[4 * q + 2] = v.z; e[4 * q + 3] = v.w;
  } else {
    if constexpr (W % 4 >= 2) {
      const uint2 v = *reinterpret_cast<const uint2 *>(row + W / 4 * 128 + lane * 2);
      e[W / 4 * 4] = v.x; e[W / 4 * 4 + 1] = v.y;
    }
    if constexpr (W % 2) e[W - 1] = row[W / 4 * 128 + (W % 4 >= 2 ? 64 : 0) + lane];
  }
}

__device__ __forceinline__ uint32_t splat16(int v) { return (uint32_t) (v & 0xffff) * 0x10001u; }
__device__ __forceinline__ int half_max(uint32_t v) { return max((int) (int16_t) (v & 0xffffu), (int) v >> 16); }

// Four words of one transition table: from registers, or from the shared copy.
template <int W, bool REG>
struct VitTrans {
  uint32_t r[REG ? kFT : 1][REG ? W : 1];
  const uint32_t *s;        // shared copy (REG false)
  __device__ __forceinline__ void group(int t, int q, int lane, uint32_t (&o)[4]) const {
    if constexpr (REG) {
#pragma unroll
      for (int e = 0; e < 4; ++e) if (4 * q + e < W) o[e] = r[t][4 * q + e];
    } else {
      const uint4 v = *reinterpret_cast<const uint4 *>(s + t * W * 32 + (q * 32 + lane) * 4);
      o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
  }
};

// Match, insert and delete cells of one row; e[] is this row's emissions and
// is refilled from next_row behind its last use.
template <int W, bool REG, bool SAT>
__device__ __forceinline__ void vitf_row(uint32_t (&Mv)[W], uint32_t (&Iv)[W], uint32_t (&Dv)[W], uint32_t (&em)[W],
                                         const VitTrans<W, REG> &T, const uint32_t *__restrict__ next_row, int lane,
                                         int xB, uint32_t F2, int &xe_out, int &dm_out) {
  constexpr int NQ = (W + 3) / 4;
  const uint32_t xBp = splat16(xB);
  uint32_t sM = __shfl_up_sync(FULL, Mv[W - 1], 1), sI = __shfl_up_sync(FULL, Iv[W - 1], 1),
           sD = __shfl_up_sync(FULL, Dv[W - 1], 1);
  if (lane == 0) sM = sI = sD = F2;
  // predecessors of word 0: the previous lane's last node, this lane's word W-1 low half
  uint32_t pM = __byte_perm(sM, Mv[W - 1], 0x5432), pI = __byte_perm(sI, Iv[W - 1], 0x5432),
           pD = __byte_perm(sD, Dv[W - 1], 0x5432);
  uint32_t xe = 0x80008000u, dmax = F2, dc = F2, sv1 = 0, dc1 = 0;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    uint32_t t[7][4];
#pragma unroll
    for (int j = 0; j < 7; ++j) T.group(j, q, lane, t[j]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int w = 4 * q + e;
      if (w >= W) break;
      const uint32_t cM = Mv[w], cI = Iv[w], cD = Dv[w];
      // the row's late values (D after its closure, xB) come last
      uint32_t sv = add_s16x2(pM, t[1][e]);
      sv = __viaddmax_s16x2(pI, t[2][e], sv);
      sv = __viaddmax_s16x2(pD, t[3][e], sv);
      sv = __viaddmax_s16x2(xBp, t[0][e], sv);
      if constexpr (SAT) {
        const uint32_t ev = em[w], en = min_s16x2(ev, 0u), ep = max_s16x2(ev, 0u);
        sv = add_s16x2(min_s16x2(max_s16x2(sv, ~add_s16x2(en, 0x7fff7fffu)), ep ^ 0x7fff7fffu), ev);
      } else {
        sv = add_s16x2(sv, em[w]);
      }
      // running maxima, one three-input maximum per two words
      if (w & 1) xe = __vimax3_s16x2(xe, sv1, sv);
      else if (w == W - 1) xe = max_s16x2(xe, sv);
      else sv1 = sv;
      Iv[w] = __viaddmax_s16x2(cI, t[6][e], __viaddmax_s16x2(cM, t[5][e], F2));
      const uint32_t mv = SAT ? max_s16x2(sv, F2) : sv;
      Mv[w] = mv;
      Dv[w] = dc;                                     // M->D from word w-1
      dc = __viaddmax_s16x2(mv, t[4][e], F2);
      if (w & 1) dmax = __vimax3_s16x2(dmax, dc1, dc);
      else if (w == W - 1) dmax = max_s16x2(dmax, dc);
      else dc1 = dc;
      pM = cM; pI = cI; pD = cD;
    }
    vitf_load<W>(em, next_row, lane, q);
  }
  uint32_t sdc = __shfl_up_sync(FULL, dc, 1);
  if (lane == 0) sdc = F2;
  Dv[0] = __byte_perm(sdc, dc, 0x5432);
  xe_out = __reduce_max_sync(FULL, half_max(xe));
  dm_out = __reduce_max_sync(FULL, half_max(dmax));
}

// D->D closure: both halves of a lane as two chains of W nodes, then a warp
// scan over the lanes' ends (bd[s]: the chain cost of the last 2^s lanes). A
// value loses at least -bmax[s] over any 2^s lanes, so the scan stops where
// even the row's largest D, dm, would end at the floor: usually before its
// first step.
template <int W, bool REG>
__device__ __forceinline__ void vitf_close(uint32_t (&Dv)[W], const VitTrans<W, REG> &T, int lane, int bl, int bh,
                                           const int (&bd)[5], const int (&bmax)[5], int F, int dm) {
  constexpr int NQ = (W + 3) / 4;
  uint32_t c = Dv[0];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    uint32_t t[4];
    T.group(7, q, lane, t);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (4 * q + e > 0 && 4 * q + e < W) { c = __viaddmax_s16x2(c, t[e], Dv[4 * q + e]); Dv[4 * q + e] = c; }
  }
  const int clo = (int) (int16_t) (c & 0xffffu), chi = (int) c >> 16;
  int end = max(chi, clo + bh);
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    if (dm + bmax[s] <= F) break;
    const int o = __shfl_up_sync(FULL, end, 1 << s);
    if (lane >= (1 << s)) end = max(end, o + bd[s]);
  }
  int vin = __shfl_up_sync(FULL, end, 1);
  if (lane == 0) vin = F;
  const int vhi = max(clo, vin + bl);
  uint32_t v = __byte_perm((uint32_t) max(vin, F), (uint32_t) max(vhi, F), 0x5410);
  // the first word tells whether anything comes in from another chain
  uint32_t t0[4];
  T.group(7, 0, lane, t0);
  const uint32_t first = __viaddmax_s16x2(v, t0[0], Dv[0]);
  if (!__any_sync(FULL, first != Dv[0])) return;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    uint32_t t[4];
    T.group(7, q, lane, t);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (4 * q + e < W) { v = __viaddmax_s16x2(v, t[e], Dv[4 * q + e]); Dv[4 * q + e] = v; }
  }
}

template <int W>
constexpr int vitf_threads() { return W <= kVitFastRegW ? 64 : 128; }

template <int W>
__global__ void __launch_bounds__(vitf_threads<W>())
vit_fast_kernel(VitFastDev V, DbDev db, const int64_t *__restrict__ slots, const int64_t *__restrict__ order,
                int64_t nids, int *__restrict__ out_xc, uint8_t *__restrict__ out_st,
                unsigned long long *__restrict__ ticket) {
  constexpr bool REG = W <= kVitFastRegW;
  extern __shared__ __align__(16) uint32_t s_trans[];
  const int lane = threadIdx.x & 31;
  VitTrans<W, REG> T;
  T.s = s_trans;
  if constexpr (REG) {
#pragma unroll
    for (int t = 0; t < kFT; ++t)
#pragma unroll
      for (int q = 0; q < (W + 3) / 4; ++q) vitf_load<W>(T.r[t], V.trans + t * W * 32, lane, q);
  } else {
    for (int i = threadIdx.x; i < kFT * W * 8; i += blockDim.x)
      reinterpret_cast<uint4 *>(s_trans)[i] = __ldg(reinterpret_cast<const uint4 *>(V.trans) + i);
    __syncthreads();
  }
  // chain costs of the closure: the low and the high half, then sums over 1, 2, 4, 8, 16 lanes
  int bl = 0, bh = 0, bd[5], bmax[5];
#pragma unroll
  for (int q = 0; q < (W + 3) / 4; ++q) {
    uint32_t t[4];
    T.group(7, q, lane, t);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (4 * q + e < W) { bl += (int) (int16_t) (t[e] & 0xffffu); bh += (int) t[e] >> 16; }
  }
  int bs = bl + bh;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    bd[s] = bs;
    bmax[s] = __reduce_max_sync(FULL, lane >= (1 << s) ? bs : -0x40000000);
    const int o = __shfl_up_sync(FULL, bs, 1 << s);
    if (lane >= (1 << s)) bs += o;
  }
  for (;;) {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(ticket, 1ull);
    t = __shfl_sync(FULL, t, 0);
    if (t >= (unsigned long long) nids) break;
    const int64_t j = order[t];                       // the longest sequences first
    const int64_t s = slots[j];
    const int L = db.len[s];
    int xC = -32768, st = L > 0 ? 0 : 2;
    if (L > 0) {
      const uint32_t *sq = reinterpret_cast<const uint32_t *>(db.codes + db.start[s]);   // padded to 16 with code 29
      const int move = V.move[L];
      const int F = V.base_w + move + V.bm_min;
      const uint32_t F2 = splat16(F);
      uint32_t Mv[W], Iv[W], Dv[W], em[W];
#pragma unroll
      for (int w = 0; w < W; ++w) Mv[w] = Iv[w] = Dv[w] = F2;
      const int xN = V.base_w;
      int xB = xN + move, xJ = -32768, top = xN, top1 = xN;   // largest score up to the last row, and the one before
      uint32_t cur = __ldg(sq), nxt = L > 4 ? __ldg(sq + 1) : 0u;
      int x = cur & 0xff;
#pragma unroll
      for (int q = 0; q < (W + 3) / 4; ++q) vitf_load<W>(em, V.emit + x * W * 32, lane, q);
      for (int i = 0; i < L; ++i) {
        // the next row's residue (padding after the last one)
        // (the largest score is taken from two rows back, whose reduction is long done)
        const bool sat = top1 > V.hot || (V.low_res >> x & 1u);
        top1 = top;
        if ((i & 3) == 3) {
          cur = nxt;
          if (i + 5 < L) nxt = __ldg(sq + (i >> 2) + 2);
        } else {
          cur >>= 8;
        }
        x = i + 1 < L ? (int) (cur & 0xff) : 0;
        const uint32_t *next_row = V.emit + x * W * 32;
        int xe, dm;
        if (sat) vitf_row<W, REG, true>(Mv, Iv, Dv, em, T, next_row, lane, xB, F2, xe, dm);
        else     vitf_row<W, REG, false>(Mv, Iv, Dv, em, T, next_row, lane, xB, F2, xe, dm);
        top = max(top, xe);
        xC = (int16_t) max(xC + V.xwC_loop, xe + V.xwE_move);
        xJ = max(xJ, xe + V.xwE_loop);
        xB = max(xJ, xN) + move;
        if (dm + V.ddbound_w > xB || xe >= 32767) {
          if (xe >= 32767) { xC = 32767; st = 1; break; }   // eslERANGE
          vitf_close<W, REG>(Dv, T, lane, bl, bh, bd, bmax, F, dm);
        }
      }
    }
    if (lane == 0) { out_xc[j] = xC; out_st[j] = (uint8_t) st; }
  }
}

template <int W>
cudaError_t launch_vit_fast(const VitFastDev &V, const DbDev &db, const int64_t *ids, const int64_t *order, int64_t n,
                            int *xc, uint8_t *st, unsigned long long *ticket, int sms, cudaStream_t stream) {
  constexpr int threads = vitf_threads<W>();
  constexpr size_t smem = W <= kVitFastRegW ? 0 : (size_t) kFT * W * 32 * 4;
  auto kern = vit_fast_kernel<W>;
  static std::atomic<unsigned long long> configured{0};
  if (smem) {
    const cudaError_t e = ensure_smem_attr((const void *) kern, smem, configured);
    if (e != cudaSuccess) return e;
  }
  int per_sm = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (e != cudaSuccess) return e;
  long long grid = (long long) (per_sm < 1 ? 1 : per_sm) * sms;
  const long long need = (n + threads / 32 - 1) / (threads / 32);
  if (need < grid) grid = need < 1 ? 1 : need;
  (void) cudaGetLastError();
  kern<<<(unsigned) grid, threads, smem, stream>>>(V, db, ids, order, n, xc, st, ticket);
  return cudaGetLastError();
}

}  // namespace msvgb

#define MSVGB_INSTANTIATE_VITF(W)                                                                          \
  template cudaError_t msvgb::launch_vit_fast<W>(const msvgb::VitFastDev &, const msvgb::DbDev &,          \
                                                 const int64_t *, const int64_t *, int64_t, int *, uint8_t *, \
                                                 unsigned long long *, int, cudaStream_t);
