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
// Bound: the ALU pipe (79% busy at M = 260, 40,000 listed sequences), on which
// the fused add-maximum and the packed add run at half rate (64 lanes per clock
// and SM): nine such operations per word of two nodes, a third of a row's
// instructions at 5 words per lane. The transition costs stay in registers across
// rows (up to 16 words per lane); a row reads only its residue's emissions.
// One warp scores a sequence up to 1024 nodes; above, the 4 or 8 warps of a
// block share it: one warp with its row in registers and the transitions in
// shared memory took 5.46 ms for a call on 3,000 listed sequences at M = 2400
// (4.1 without its host work), four warps take 2.19 (2.27 with the closure's
// chains only in the rows that ask for them).
#pragma once
#include <cuda_runtime.h>

#include "msv_device.cuh"

namespace msvgb {

// Transition tables: BM MM IM DM (into the node), MD MI II (out of it), DD (into it).
constexpr int kFT = 8;

struct VitFastDev {
  int base_w, ddbound_w, xwE_move, xwE_loop, xwC_loop;
  int bm_min;               // smallest entry cost of a real node: F = base + move + bm_min
  int hot;                  // 32767 - twice the largest emission: no row can pass 32767 within the next two
  uint32_t low_res;         // residues whose emissions need the saturating row
  const uint32_t *trans;    // [kFT] rows of the lane layout below
  const uint32_t *emit;     // [NRES] rows
  const int16_t *move;      // [Lmax + 1]
};

// N lanes (32 per warp) score one sequence. One row of W words per lane,
// lane-contiguous in 16-byte quads [q][N][4], then a pair [N][2] and a single
// [N] for the remainder: W * N words. Word w of lane l holds nodes
// l * 2W + w + 1 (low half) and l * 2W + W + w + 1.
__host__ __device__ constexpr int vitf_at(int W, int N, int lane, int w) {
  return w < W / 4 * 4 ? (w / 4 * N + lane) * 4 + w % 4
       : (W % 4 >= 2 && w < W / 4 * 4 + 2) ? W / 4 * 4 * N + lane * 2 + (w - W / 4 * 4)
                                           : W / 4 * 4 * N + (W % 4 >= 2 ? 2 * N : 0) + lane;
}

// Words 4q .. 4q+3 of a row (the last call of a row takes the remainder).
template <int W, int N>
__device__ __forceinline__ void vitf_load(uint32_t (&e)[W], const uint32_t *__restrict__ row, int lane, int q) {
  if (q < W / 4) {
    const uint4 v = *reinterpret_cast<const uint4 *>(row + (q * N + lane) * 4);
    e[4 * q] = v.x; e[4 * q + 1] = v.y; e[4 * q + 2] = v.z; e[4 * q + 3] = v.w;
  } else {
    if constexpr (W % 4 >= 2) {
      const uint2 v = *reinterpret_cast<const uint2 *>(row + W / 4 * 4 * N + lane * 2);
      e[W / 4 * 4] = v.x; e[W / 4 * 4 + 1] = v.y;
    }
    if constexpr (W % 2) e[W - 1] = row[W / 4 * 4 * N + (W % 4 >= 2 ? 2 * N : 0) + lane];
  }
}

__device__ __forceinline__ uint32_t splat16(int v) { return (uint32_t) (v & 0xffff) * 0x10001u; }
__device__ __forceinline__ int half_max(uint32_t v) { return max((int) (int16_t) (v & 0xffffu), (int) v >> 16); }

// Match, insert and delete cells of one row from the predecessors of this
// lane's word 0 (pM, pI, pD); em[] is this row's emissions and is refilled from
// next_row behind its last use. Dv[0] is left to the caller; dc_out is the
// M->D of the last word. xe and dmax: this lane's maxima.
template <int W, int N, bool SAT>
__device__ __forceinline__ void vitf_row(uint32_t (&Mv)[W], uint32_t (&Iv)[W], uint32_t (&Dv)[W], uint32_t (&em)[W],
                                         const uint32_t (&T)[kFT][W], const uint32_t *__restrict__ next_row, int lane,
                                         int xB, uint32_t F2, uint32_t pM, uint32_t pI, uint32_t pD, uint32_t &dc_out,
                                         int &xe_out, int &dm_out) {
  const uint32_t xBp = splat16(xB);
  uint32_t xe = 0x80008000u, dmax = F2, dc = F2, sv1 = 0, dc1 = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const uint32_t cM = Mv[w], cI = Iv[w], cD = Dv[w];
    // the row's late values (D after its closure, xB) come last
    uint32_t sv = add_s16x2(pM, T[1][w]);
    sv = __viaddmax_s16x2(pI, T[2][w], sv);
    sv = __viaddmax_s16x2(pD, T[3][w], sv);
    sv = __viaddmax_s16x2(xBp, T[0][w], sv);
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
    Iv[w] = __viaddmax_s16x2(cI, T[6][w], __viaddmax_s16x2(cM, T[5][w], F2));
    const uint32_t mv = SAT ? max_s16x2(sv, F2) : sv;
    Mv[w] = mv;
    Dv[w] = dc;                                       // M->D from word w-1
    dc = __viaddmax_s16x2(mv, T[4][w], F2);
    if (w & 1) dmax = __vimax3_s16x2(dmax, dc1, dc);
    else if (w == W - 1) dmax = max_s16x2(dmax, dc);
    else dc1 = dc;
    pM = cM; pI = cI; pD = cD;
    if (w % 4 == 3 || w == W - 1) vitf_load<W, N>(em, next_row, lane, w / 4);
  }
  dc_out = dc;
  xe_out = half_max(xe);
  dm_out = half_max(dmax);
}

// Chain costs of the D->D closure: the low and the high half of a lane, sums
// over the warp's last 1, 2, 4, 8, 16 lanes (bd) with their largest over the
// lanes (bmax), and over the warp's lanes before this one (pre).
struct VitChains {
  int bl, bh, bd[5], bmax[5], pre;
};
template <int W>
__device__ __forceinline__ void vitf_chains(const uint32_t (&dd)[W], int lane, VitChains &c) {
  c.bl = c.bh = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) { c.bl += (int) (int16_t) (dd[w] & 0xffffu); c.bh += (int) dd[w] >> 16; }
  int bs = c.bl + c.bh;
  const int own = bs;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    c.bd[s] = bs;
    c.bmax[s] = __reduce_max_sync(FULL, lane >= (1 << s) ? bs : -0x40000000);
    const int o = __shfl_up_sync(FULL, bs, 1 << s);
    if (lane >= (1 << s)) bs += o;
  }
  c.pre = bs - own;
}

// The closure: both halves of a lane as two chains of W nodes; end: the value
// leaving the lane, from within it. Where the warps of a block share a
// sequence the chains run in every row, beside the maxima's reductions, whose
// exchange the row waits for anyway (a D closed where the bound does not ask
// for it changes nothing); a warp on its own runs them only where asked.
template <int W>
__device__ __forceinline__ int vitf_chain(uint32_t (&Dv)[W], const uint32_t (&dd)[W], const VitChains &ch, int &clo) {
  uint32_t c = Dv[0];
#pragma unroll
  for (int w = 1; w < W; ++w) { c = __viaddmax_s16x2(c, dd[w], Dv[w]); Dv[w] = c; }
  clo = (int) (int16_t) (c & 0xffffu);
  return max((int) c >> 16, clo + ch.bh);
}

// A warp scan of the lanes' ends, for rows whose largest D, dm, lives through
// a lane's chains: a value loses at least -bmax[s] over any 2^s lanes, and the
// scan stops where even dm would end at the floor.
__device__ __forceinline__ int vitf_scan(int end, int lane, const VitChains &ch, int F, int dm) {
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    if (dm + ch.bmax[s] <= F) break;
    const int o = __shfl_up_sync(FULL, end, 1 << s);
    if (lane >= (1 << s)) end = max(end, o + ch.bd[s]);
  }
  return end;
}

// Runs the value vin coming into the lane through both of its chains.
template <int W>
__device__ __forceinline__ void vitf_apply(uint32_t (&Dv)[W], const uint32_t (&dd)[W], const VitChains &ch, int F,
                                           int vin, int clo) {
  uint32_t v = __byte_perm((uint32_t) max(vin, F), (uint32_t) max(max(clo, vin + ch.bl), F), 0x5410);
  // the first word tells whether anything comes in from another chain
  const uint32_t first = __viaddmax_s16x2(v, dd[0], Dv[0]);
  if (!__any_sync(FULL, first != Dv[0])) return;
#pragma unroll
  for (int w = 0; w < W; ++w) { v = __viaddmax_s16x2(v, dd[w], Dv[w]); Dv[w] = v; }
}

// One sequence of the list, NW warps: NW = 1, a warp on its own; else the
// block's warps share it, exchanging their last lanes' cells and their maxima
// through shared memory (two barriers a row, three with a closure).
template <int NW>
struct VitShared {
  uint32_t M[2][NW], I[2][NW], D[NW], dc[NW];         // last lanes; M, I of the row's parity
  int xe[NW], dm[NW], end[NW], sum[NW];               // maxima, closure ends, chain cost of the whole warp
  unsigned long long t;
};

template <int W, int NW>
__global__ void __launch_bounds__(NW == 1 ? 64 : NW * 32)
vit_fast_kernel(VitFastDev V, DbDev db, const int64_t *__restrict__ slots, const int64_t *__restrict__ order,
                int64_t nids, int *__restrict__ out_xc, uint8_t *__restrict__ out_st,
                unsigned long long *__restrict__ ticket) {
  constexpr int N = 32 * NW;
  __shared__ VitShared<NW> sh;
  const int lane = threadIdx.x & 31, warp = NW == 1 ? 0 : threadIdx.x >> 5, vlane = warp * 32 + lane;
  uint32_t T[kFT][W];
#pragma unroll
  for (int t = 0; t < kFT; ++t)
#pragma unroll
    for (int q = 0; q < (W + 3) / 4; ++q) vitf_load<W, N>(T[t], V.trans + t * W * N, vlane, q);
  VitChains ch;
  vitf_chains<W>(T[7], lane, ch);
  if (NW > 1 && lane == 31) sh.sum[warp] = ch.pre + ch.bl + ch.bh;
  for (;;) {
    unsigned long long t = 0;
    if constexpr (NW == 1) {
      if (lane == 0) t = atomicAdd(ticket, 1ull);
      t = __shfl_sync(FULL, t, 0);
    } else {
      __syncthreads();                                // the last sequence is done with sh
      if (threadIdx.x == 0) sh.t = atomicAdd(ticket, 1ull);
      __syncthreads();
      t = sh.t;
    }
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
      for (int q = 0; q < (W + 3) / 4; ++q) vitf_load<W, N>(em, V.emit + x * W * N, vlane, q);
      for (int i = 0; i < L; ++i) {
        // (the largest score is taken from two rows back, whose reduction is long done)
        const bool sat = top1 > V.hot || (V.low_res >> x & 1u);
        top1 = top;
        // the next row's residue
        if ((i & 3) == 3) {
          cur = nxt;
          if (i + 5 < L) nxt = __ldg(sq + (i >> 2) + 2);
        } else {
          cur >>= 8;
        }
        x = i + 1 < L ? (int) (cur & 0xff) : 0;
        const uint32_t *next_row = V.emit + x * W * N;
        // predecessors of word 0: the previous lane's last node, this lane's word W-1 low half
        uint32_t sM = __shfl_up_sync(FULL, Mv[W - 1], 1), sI = __shfl_up_sync(FULL, Iv[W - 1], 1),
                 sD = __shfl_up_sync(FULL, Dv[W - 1], 1);
        if (lane == 0) {
          sM = sI = sD = F2;
          if (NW > 1 && warp > 0 && i > 0) { sM = sh.M[i & 1][warp - 1]; sI = sh.I[i & 1][warp - 1]; sD = sh.D[warp - 1]; }
        }
        const uint32_t pM = __byte_perm(sM, Mv[W - 1], 0x5432), pI = __byte_perm(sI, Iv[W - 1], 0x5432),
                       pD = __byte_perm(sD, Dv[W - 1], 0x5432);
        uint32_t dc;
        int xe, dm;
        if (sat) vitf_row<W, N, true>(Mv, Iv, Dv, em, T, next_row, vlane, xB, F2, pM, pI, pD, dc, xe, dm);
        else     vitf_row<W, N, false>(Mv, Iv, Dv, em, T, next_row, vlane, xB, F2, pM, pI, pD, dc, xe, dm);
        xe = __reduce_max_sync(FULL, xe);
        dm = __reduce_max_sync(FULL, dm);
        uint32_t sdc = __shfl_up_sync(FULL, dc, 1);
        if (lane == 0) sdc = F2;
        if constexpr (NW > 1) {
          if (lane == 31) {
            sh.M[~i & 1][warp] = Mv[W - 1]; sh.I[~i & 1][warp] = Iv[W - 1];
            sh.dc[warp] = dc; sh.xe[warp] = xe; sh.dm[warp] = dm;
          }
          __syncthreads();
          if (lane == 0 && warp > 0) sdc = sh.dc[warp - 1];
#pragma unroll
          for (int k = 0; k < NW; ++k) { xe = max(xe, sh.xe[k]); dm = max(dm, sh.dm[k]); }
        }
        Dv[0] = __byte_perm(sdc, dc, 0x5432);
        int clo = 0, end = 0, vin = F, into = F;
        if constexpr (NW > 1) {
          end = vitf_chain<W>(Dv, T[7], ch, clo);
          vin = __shfl_up_sync(FULL, end, 1);
        }
        top = max(top, xe);
        xC = (int16_t) max(xC + V.xwC_loop, xe + V.xwE_move);
        xJ = max(xJ, xe + V.xwE_loop);
        xB = max(xJ, xN) + move;
        if (dm + V.ddbound_w > xB || xe >= 32767) {
          if (xe >= 32767) { xC = 32767; st = 1; break; }   // eslERANGE
          if constexpr (NW == 1) end = vitf_chain<W>(Dv, T[7], ch, clo);
          if (NW == 1 || dm + ch.bmax[0] > F) {
            end = vitf_scan(end, lane, ch, F, dm);
            vin = __shfl_up_sync(FULL, end, 1);
          }
          if constexpr (NW > 1) {                     // the earlier warps' ends, carried through the warps between
            if (lane == 31) sh.end[warp] = end;
            __syncthreads();
            for (int k = 0; k < warp; ++k) into = max(sh.end[k], into + sh.sum[k]);
          }
          vin = lane == 0 ? into : NW > 1 ? max(vin, into + ch.pre) : vin;
          vitf_apply<W>(Dv, T[7], ch, F, vin, clo);
        }
        if constexpr (NW > 1) {
          if (lane == 31) sh.D[warp] = Dv[W - 1];
          __syncthreads();
        }
      }
    }
    if (vlane == 0) { out_xc[j] = xC; out_st[j] = (uint8_t) st; }
  }
}

template <int W, int NW>
cudaError_t launch_vit_fast(const VitFastDev &V, const DbDev &db, const int64_t *ids, const int64_t *order, int64_t n,
                            int *xc, uint8_t *st, unsigned long long *ticket, int sms, cudaStream_t stream) {
  constexpr int threads = NW == 1 ? 64 : NW * 32, per_block = threads / 32 / NW;
  auto kern = vit_fast_kernel<W, NW>;
  int per_sm = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, 0);
  if (e != cudaSuccess) return e;
  long long grid = (long long) (per_sm < 1 ? 1 : per_sm) * sms;
  const long long need = (n + per_block - 1) / per_block;
  if (need < grid) grid = need < 1 ? 1 : need;
  (void) cudaGetLastError();
  kern<<<(unsigned) grid, threads, 0, stream>>>(V, db, ids, order, n, xc, st, ticket);
  return cudaGetLastError();
}

}  // namespace msvgb

#define MSVGB_INSTANTIATE_VITF(W, NW)                                                                      \
  template cudaError_t msvgb::launch_vit_fast<W, NW>(const msvgb::VitFastDev &, const msvgb::DbDev &,          \
                                                 const int64_t *, const int64_t *, int64_t, int *, uint8_t *, \
                                                 unsigned long long *, int, cudaStream_t);
