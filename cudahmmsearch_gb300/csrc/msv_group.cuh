// msv_group.cuh -- SSV pass with G < 32 lanes per sequence.
//
// For small models a whole warp per sequence leaves each lane only a few DP
// words per row, so the per-row overhead (the shuffle, the residue decode,
// the table address) dominates. Here G lanes (4, 8 or 16; 32 for models of 1024
// nodes and more) score one sequence and a warp carries 32/G sequences in
// lockstep: each group owns its sequence
// state (index, row, residue word) and fetches the next sequence when its own
// ends, while all lanes execute the same row code every step (finished groups
// run pad rows, whose costs keep every cell at the floor). Lane g of a group
// owns nodes g*2C+1 .. (g+1)*2C with the same two-way striping as the 32-lane
// kernel. Only phase A (SSV) runs here; sequences SSV leaves undecided, or
// whose length disables SSV, are appended to a list that the same lane groups
// then score with the full MSV recurrence (msv_list_group_kernel).
#pragma once
#include "msv_device.cuh"

namespace msvgb {

// Copies of the table regions. A shared-memory access is served in phases of
// 128 bytes (8 lanes for 16-byte loads, 16 for 8-byte, 32 for 4-byte loads);
// where one phase holds several groups (16-byte loads at 4 lanes per group,
// 8-byte loads at 8 or fewer, 4-byte loads at 16 or fewer), each reading its
// own residue's row, two rows whose offsets meet on the same banks conflict.
// Those regions are therefore stored once per group of a phase, each copy on
// its own banks: group j of the phase reads copy j.
template <int G> struct GroupCopies {
  static constexpr int QUAD = G < 8 ? 8 / G : 1;          // 16-byte loads: groups per 8 lanes
  static constexpr int PAIR = G < 16 ? 16 / G : 1;       // 8-byte loads: groups per 16 lanes
  static constexpr int SINGLE = 32 / G;                   // 4-byte loads: groups per warp
};

template <int C, int G>
struct GroupLayout {
  static constexpr int Q4 = C / 4, R = C % 4;
  static constexpr int A_WORDS = NRES * Q4 * GroupCopies<G>::QUAD * G * 4;             // quads [x][q][copy][g][4]
  static constexpr int B_WORDS = (R >= 2) ? NRES * GroupCopies<G>::PAIR * G * 2 : 0;   // pair  [x][copy][g][2]
  static constexpr int C_WORDS = (R & 1) ? NRES * GroupCopies<G>::SINGLE * G : 0;      // single [x][copy][g]
  static constexpr int WORDS = A_WORDS + B_WORDS + C_WORDS;
};

template <int C, int G>
__device__ __forceinline__ void ssv_row_group(uint32_t (&dp)[C], uint32_t &acc0, uint32_t &acc1,
                                              const uint32_t *__restrict__ tab, int x, int glane, int gidx,
                                              int src_lane) {
  using Lay = GroupLayout<C, G>;
  using Cp = GroupCopies<G>;
  constexpr uint32_t one2 = 0x3C003C00u;
  uint32_t s[C];
#pragma unroll
  for (int q = 0; q < Lay::Q4; ++q) {
    const uint4 v = *reinterpret_cast<const uint4 *>(tab + (((x * Lay::Q4 + q) * Cp::QUAD + gidx % Cp::QUAD) * G + glane) * 4);
    s[4 * q] = v.x; s[4 * q + 1] = v.y; s[4 * q + 2] = v.z; s[4 * q + 3] = v.w;
  }
  if constexpr (Lay::R >= 2) {
    const int cp = gidx % Cp::PAIR;
    const uint2 v = *reinterpret_cast<const uint2 *>(tab + Lay::A_WORDS + ((x * Cp::PAIR + cp) * G + glane) * 2);
    s[4 * Lay::Q4] = v.x; s[4 * Lay::Q4 + 1] = v.y;
  }
  if constexpr (Lay::R & 1) s[C - 1] = tab[Lay::A_WORDS + Lay::B_WORDS + (x * Cp::SINGLE + gidx) * G + glane];
  const uint32_t pred0 = pred_word0(dp[C - 1], src_lane);   // all 32 lanes, every row
#pragma unroll
  for (int w = C - 1; w >= 0; --w) dp[w] = fma_relu_f16x2(w ? dp[w - 1] : pred0, one2, s[w]);
  // the running maximum on the bits (non-negative f16 order like signed
  // integers), one three-input maximum per two words as in ssv_row_hyb
  if constexpr (C & 1) acc1 = max_s16x2(acc1, dp[C - 1]);
#pragma unroll
  for (int w = 0; w + 1 < C; w += 2) acc0 = __vimax3_s16x2(acc0, dp[w], dp[w + 1]);
}

// ---- mixed-width SSV table (f16 and 8-bit costs) ------------------------------
// The f16 row reads 2 bytes of cost per cell from shared memory and is bound
// by shared-memory bandwidth (one 128-byte wavefront per clock and SM) while
// the FMA and ALU pipes idle half the time. Here the last CI words of every
// lane keep their costs as bytes (1 byte per cell) and widen them in
// registers, trading shared-memory bytes for instructions on the idle pipes.
//
// Units: cells and f16 costs are integers times 2^-24, i.e. f16 subnormals
// (and the smallest normals): an integer n with |n| < 2048 is exact, and the
// bits of a cell (n >= 0) are the 16-bit integer n itself (a cost n < 0 is
// 0x8000 | -n). So a cell is an f16 and an integer at once, and each word
// takes whichever update suits the pipes: f16 words one fma.relu (FMA pipe);
// 8-bit words either one PRMT that sign-extends the byte and one integer
// add-and-maximum max(u + s, 0) (both on the ALU pipe), or, where the ALU pipe
// with the running maximum on it is the fuller one, one PRMT to the f16 t =
// s + 128, one f16 add of -128 and the fma.relu (hyb_biased of the words; their
// bytes hold t). All are exact for the same reason. Bits order like signed
// 16-bit integers, so the running maximum is taken on the bits too.
//
// Layout for residue x (CF = C - CI f16 words, CI a multiple of 4): the f16
// regions of GroupLayout<CF, G> (quads, pair, single), then 16-byte octets
// [x][o][copy][g][4 words], then, when CI % 8 == 4, one 8-byte half octet
// [x][copy][g][2 words] (copies as GroupCopies): word k of octet o of lane g holds the bytes
// [s(w, h0), s(w+1, h0), s(w, h1), s(w+1, h1)] of DP words w = CF + 8o + 2k
// and w + 1 (the half octet: w = CF + 8 * NO + 2k).
__device__ __forceinline__ uint32_t add_f16x2(uint32_t a, uint32_t b) {
  uint32_t d; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d;
}
// Default 8-bit words per lane of the G-lane SSV pass at DP width C, and how
// many of them take the FMA pipe, from a sweep on GB300 (TCUPS with 0 / 4 / 8 /
// 12 words; 800,000 sequences at 8 lanes, 400,000 at 16, 250,000 at 32; a: 4 of
// the words on the FMA pipe): C = 10: 13.4 / 14.3a; 12: 14.0 / 15.6 / 14.1a;
// 16: 15.2 / 16.7 / 16.7a; 18: 15.6 / 16.9 / 17.3a; 22: 15.7 / 17.2 / 18.0a;
// 24: 16.2 / 17.4 / 18.8; 28: 16.0 / - / 18.5 / 19.0a; 32: 16.9 / - / 18.8 / 19.5a;
// 16 lanes: C = 20: 16.6 / 18.1 / 19.1a; 24: 16.9 / 16.9 / 19.6; 32: 17.5 / 17.5 /
// 19.6 / 20.4a; 32 lanes: C = 17: - / 18.4 / 18.6a; 24: - / 18.6 / 20.1; 32: - /
// 19.1 / 20.3 / 20.9a. With every 8-bit word on the FMA pipe C = 26 took 16.3 ms
// for 2,000,000 sequences, 15.8 with none. At C = 26 and 8 words the pass reads
// shared memory in 97.7% of cycles, but more 8-bit words still lose below 28
// (12 with 4 on the FMA pipe: 18.3, 16 with 8: 18.5, 8: 19.5): the ALU pipe takes
// over; 12 with none there was not measured. 4 lanes take the 8-lane shares,
// unswept.
__host__ __device__ constexpr int hyb_words(int C, int G) {
  if (G == 32) return C < 17 ? 0 : 8;
  if (C < (G == 16 ? 13 : 10)) return 0;
  return C < 18 ? 4 : C < 28 ? 8 : 12;
}
__host__ __device__ constexpr int hyb_biased(int C, int CI) { return CI == 4 ? (C < 12 ? 4 : 0) : CI == 8 && C >= 24 ? 0 : 4; }

template <int C, int CI, int G>
struct HybLayout {
  static_assert(CI % 4 == 0 && CI >= 4 && CI <= C, "8-bit words come in fours");
  static constexpr int CF = C - CI, CB = CF + hyb_biased(C, CI);   // words below CB run on the FMA pipe
  static constexpr int Q4 = CF / 4, R = CF % 4, NO = CI / 8, HALF = (CI % 8) / 4;
  static constexpr int A_WORDS = NRES * Q4 * GroupCopies<G>::QUAD * G * 4;
  static constexpr int B_WORDS = (R >= 2) ? NRES * GroupCopies<G>::PAIR * G * 2 : 0;
  static constexpr int C_WORDS = (R & 1) ? NRES * GroupCopies<G>::SINGLE * G : 0;
  static constexpr int D_WORDS = NRES * NO * GroupCopies<G>::QUAD * G * 4;
  static constexpr int E_WORDS = NRES * HALF * GroupCopies<G>::PAIR * G * 2;   // [x][copy][g][2]
  static constexpr int WORDS = A_WORDS + B_WORDS + C_WORDS + D_WORDS + E_WORDS;
};

// The costs of two 8-bit words from a table word's bytes: as f16 (t - 128
// units), or as sign-extended integers.
__device__ __forceinline__ void hyb_widen(uint32_t t, bool f16, uint32_t &a, uint32_t &b) {
  constexpr uint32_t m128 = 0x80808080u;        // f16x2 (-128, -128) units of 2^-24
  a = f16 ? add_f16x2(prmt(t, 0u, 0x4240u), m128) : prmt(t, 0u, 0xA280u);   // bytes 0, 2
  b = f16 ? add_f16x2(prmt(t, 0u, 0x4341u), m128) : prmt(t, 0u, 0xB391u);   // bytes 1, 3
}

template <int C, int CI, int G>
__device__ __forceinline__ void ssv_row_hyb(uint32_t (&dp)[C], uint32_t &acc0, uint32_t &acc1,
                                            const uint32_t *__restrict__ tab, int x, int glane, int gidx,
                                            int src_lane) {
  using Lay = HybLayout<C, CI, G>;
  using Cp = GroupCopies<G>;
  constexpr int CF = Lay::CF;
  constexpr uint32_t one2 = 0x3C003C00u;        // f16x2 (1.0, 1.0)
  uint32_t s[C];
#pragma unroll
  for (int q = 0; q < Lay::Q4; ++q) {
    const uint4 v = *reinterpret_cast<const uint4 *>(tab + (((x * Lay::Q4 + q) * Cp::QUAD + gidx % Cp::QUAD) * G + glane) * 4);
    s[4 * q] = v.x; s[4 * q + 1] = v.y; s[4 * q + 2] = v.z; s[4 * q + 3] = v.w;
  }
  if constexpr (Lay::R >= 2) {
    const int cp = gidx % Cp::PAIR;
    const uint2 v = *reinterpret_cast<const uint2 *>(tab + Lay::A_WORDS + ((x * Cp::PAIR + cp) * G + glane) * 2);
    s[4 * Lay::Q4] = v.x; s[4 * Lay::Q4 + 1] = v.y;
  }
  if constexpr (Lay::R & 1) s[CF - 1] = tab[Lay::A_WORDS + Lay::B_WORDS + (x * Cp::SINGLE + gidx) * G + glane];
  const uint32_t *td = tab + Lay::A_WORDS + Lay::B_WORDS + Lay::C_WORDS;
#pragma unroll
  for (int o = 0; o < Lay::NO; ++o) {
    const uint4 v = *reinterpret_cast<const uint4 *>(td + (((x * Lay::NO + o) * Cp::QUAD + gidx % Cp::QUAD) * G + glane) * 4);
    const uint32_t tw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      hyb_widen(tw[k], CF + 8 * o + 2 * k < Lay::CB, s[CF + 8 * o + 2 * k], s[CF + 8 * o + 2 * k + 1]);
    }
  }
  if constexpr (Lay::HALF) {
    const int cp = gidx % Cp::PAIR;
    const uint2 v = *reinterpret_cast<const uint2 *>(td + Lay::D_WORDS + ((x * Cp::PAIR + cp) * G + glane) * 2);
    const uint32_t tw[2] = {v.x, v.y};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      hyb_widen(tw[k], CF + 8 * Lay::NO + 2 * k < Lay::CB, s[CF + 8 * Lay::NO + 2 * k], s[CF + 8 * Lay::NO + 2 * k + 1]);
    }
  }
  const uint32_t pred0 = pred_word0(dp[C - 1], src_lane);
#pragma unroll
  for (int w = C - 1; w >= 0; --w)
    dp[w] = w < Lay::CB ? fma_relu_f16x2(w ? dp[w - 1] : pred0, one2, s[w])
                   : __viaddmax_s16x2(w ? dp[w - 1] : pred0, s[w], 0u);
  // running maximum on the bits (non-negative; fma.rn.relu gives +0, never -0,
  // which the integer words would read as -32768: all 2048 x 511 pairs of a
  // cell and a cost checked on the GPU):
  // one three-input maximum per two words takes fewer issue slots than two
  // maxima, and issue, not the integer pipe, is what this row runs short of
  // (measured: 16.3 vs 17.0 ms at M = 400 on 2,000,000 sequences)
  if constexpr (C & 1) acc1 = max_s16x2(acc1, dp[C - 1]);
#pragma unroll
  for (int w = 0; w + 1 < C; w += 2) acc0 = __vimax3_s16x2(acc0, dp[w], dp[w + 1]);
}

// The group maximum of a hybrid accumulator as a float number of units
// (capped at 4096: above 2047 units values are not exact, and past the trust
// bound only "large" matters).
__device__ __forceinline__ float hyb_units(uint32_t acc) {
  const int lo = (int) (int16_t) (acc & 0xFFFFu), hi = (int) (int16_t) (acc >> 16);
  const int b = max(max(lo, hi), 0);
  if (b >= 0x7C00) return 4096.0f;                         // inf: far past any bound
  const float f = __half2float(__ushort_as_half((unsigned short) b)) * 16777216.0f;
  return fminf(f, 4096.0f);
}

struct GroupArgs {
  ProfDev P;                       // P.stab: the G-lane f16 SSV table
  DbDev db;
  uint8_t *out_xj, *out_flags;
  unsigned long long *ticket;
  int64_t *undecided;              // sorted indices left for the full MSV pass
  unsigned long long *n_undecided;
  int64_t s_begin = 0;             // first sorted sequence of the pass (the rest of the database follows)
  SegDev segs{};                   // segments of the longest sequences (s_begin 0)
  cudaStream_t stream;
};

constexpr int64_t kSegItem = (int64_t) 1 << 62;
constexpr uint32_t kPadWord = 0x1D1D1D1Du;   // four PAD_CODE residues

// The lockstep SSV loop of one warp. fetch() (called by lane 0 of a group)
// returns the next sorted sequence index, or a negative value when there is
// none; undecided(s) (lane 0 of a group) records a sequence that needs the full
// MSV. Decided sequences (and empty ones) are written to out_xj / out_flags.
// CI > 0: the mixed-width table (HybLayout<C, CI, G>, units of 2^-24). SEG:
// fetch() returns a work item, the segments of segs first.
template <int C, int G, int CI = 0, bool SEG = false, class Fetch, class Undecided>
__device__ __forceinline__ void ssv_group_loop(const ProfDev &P, const uint32_t *__restrict__ tab, const DbDev &db,
                                               uint8_t *__restrict__ out_xj, uint8_t *__restrict__ out_flags,
                                               Fetch fetch, Undecided undecided, const SegDev &segs = SegDev()) {
  const int lane = threadIdx.x & 31, glane = lane % G, gbase = lane - glane, gidx = lane / G;
  const int src_lane = gbase + (glane + G - 1) % G;
  const unsigned gmask = (G == 32) ? FULL : (((1u << G) - 1u) << gbase);
  const int tbm = P.tbm, tec = P.tec, base = P.base, bias = P.bias;

  int64_t s = 0;                                      // SEG: kSegItem | work item while the group scores a segment
  int L = 0, i = 0;                                   // L: where the item's rows (SEG: the block's) end
  const uint2 *sq = nullptr;
  uint2 nextw = make_uint2(kPadWord, kPadWord);
  bool need = true, done = false;
  uint32_t dp[C];
  uint32_t acc0 = 0u, acc1 = 0u;
#pragma unroll
  for (int w = 0; w < C; ++w) dp[w] = 0u;

  for (;;) {
    if (need && !done) {                              // group-uniform: take the next sequence
      long long t = 0;
      if (glane == 0) t = fetch();
      t = __shfl_sync(gmask, t, gbase);
      if (t < 0) {
        done = true;
      } else {
        s = (int64_t) t;
        int k = -1;                                   // segment index
        if constexpr (SEG) {
          const long long nseg = segs.base[segs.S];
          if (t < nseg) { k = seg_of(segs, (uint32_t) t); s = t - segs.base[k]; }
          else s = t - nseg + segs.nl;
        }
        L = db.len[s];
        const int tjb = P.tjb[L];
        if (SEG && k >= 0) {
          sq = reinterpret_cast<const uint2 *>(db.codes + db.start[s]);
          i = max(0, k * segs.T - segs.warm);
          L = min(L, k * segs.T + segs.R);
          s = kSegItem | t;
          nextw = __ldg(sq + (i >> 3));
          need = false;
#pragma unroll
          for (int w = 0; w < C; ++w) dp[w] = 0u;
          acc0 = acc1 = 0u;
        } else if (L == 0) {                                 // skipped, as p7_Pipeline does
          if (glane == 0) { const int64_t oi = db.orig[s]; out_xj[oi] = 0; out_flags[oi] = 0x08; }
        } else if (tjb + tbm + tec + bias >= 127) {   // SSV disabled for this length: full MSV
          if (glane == 0) undecided(s);
        } else {
          sq = reinterpret_cast<const uint2 *>(db.codes + db.start[s]);
          nextw = __ldg(sq);
          i = 0;
          need = false;
#pragma unroll
          for (int w = 0; w < C; ++w) dp[w] = 0u;
          acc0 = acc1 = 0u;
        }
      }
    }
    if (__all_sync(FULL, done)) break;
    const bool active = !need && !done;
    // eight rows a step (sequences are padded to 16)
    const uint32_t w8[2] = {active ? nextw.x : kPadWord, active ? nextw.y : kPadWord};
    if (active && (SEG || i + 8 < L)) nextw = __ldg(sq + (i >> 3) + 1);   // SEG: may run into the buffer's padding
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int x = (w8[j >> 2] >> (8 * (j & 3))) & 0xFF;
      if constexpr (CI > 0) ssv_row_hyb<C, CI, G>(dp, acc0, acc1, tab, x, glane, gidx, src_lane);
      else                  ssv_row_group<C, G>(dp, acc0, acc1, tab, x, glane, gidx, src_lane);
    }
    i += 8;
    const bool fin = active && i >= L;
    if (__any_sync(FULL, fin)) {                      // group maxima (all lanes take part)
      float f;
      if constexpr (CI > 0) {
        f = hyb_units(max_s16x2(acc0, acc1));
      } else {
        const __half2 a = __hmax2(*reinterpret_cast<const __half2 *>(&acc0),
                                  *reinterpret_cast<const __half2 *>(&acc1));
        f = fminf(fmaxf(__low2float(a), __high2float(a)), 4096.0f);
      }
#pragma unroll
      for (int off = G / 2; off >= 1; off >>= 1) f = fmaxf(f, __shfl_xor_sync(FULL, f, off));
      if (fin) {
        int xj = 0, umax = (int) f;
        need = true;
        if (SEG && (s & kSegItem)) {                  // a segment's block
          const uint32_t item = (uint32_t) (s & ~kSegItem);
          const int k = seg_of(segs, item);
          const int64_t slot = item - segs.base[k];
          const int len = db.len[slot], end = min(len, (k + 1) * segs.T);
          if (glane == 0) segs.u[slot * segs.NB + (L - 1) / segs.R] = (uint8_t) min(umax, 255);
          if (L < end) {
            L = min(end, L + segs.R);
            acc0 = acc1 = 0u;
            need = false;
          } else if (glane == 0) {                    // the sequence's last segment to finish decides it
            s = slot;
            L = len;
            umax = seg_finish(segs, slot, len);
          }
        }
        if (need && glane == 0 && umax >= 0) {
          const int tjb = P.tjb[L];
          const int st = tjb + tbm + tec + bias < 127 ? ssv_decide(umax, tjb, tbm, tec, base, bias, xj) : -1;
          if (st < 0) {
            undecided(s);
          } else {
            const int64_t oi = db.orig[s];
            int flags = 0;
            if (st == ST_ERANGE) flags |= 0x01 | 0x02;
            else if (xj >= P.xjmin[L]) flags |= 0x02;
            out_xj[oi] = (uint8_t) xj;
            out_flags[oi] = (uint8_t) flags;
          }
        }
      }
    }
  }
}

// Stand-alone SSV pass over the sorted sequences [s_begin, n) (global
// ticket); undecided sequences go to a global list for the full-MSV launch.
// Table words of a lane-group SSV table at run-time (Cg, G, CI): the layouts
// above (GroupLayout, or HybLayout when CI > 0) with their region copies.
__host__ __device__ constexpr int group_words(int Cg, int G, int CI) {
  const int quad = G < 8 ? 8 / G : 1, pair = G < 16 ? 16 / G : 1;    // GroupCopies
  return NRES * G * ((Cg - CI) / 4 * 4 * quad + ((Cg - CI) % 4 >= 2 ? 2 * pair : 0) +
                     (((Cg - CI) % 4) & 1 ? 32 / G : 0) + CI / 8 * 4 * quad + ((CI % 8) / 4) * 2 * pair);
}

// Table words of the lane-group SSV pass: f16 (CI = 0) or mixed width.
template <int C, int G, int CI>
__host__ __device__ constexpr int group_table_words() {
  if constexpr (CI > 0) return HybLayout<C, CI, G>::WORDS;
  else return GroupLayout<C, G>::WORDS;
}

// Blocks per SM the pass is compiled for (0: the compiler's own choice). Without
// segments a bound of one, which frees the registers to load costs further
// ahead, is the faster below 24 words and at 28: us at 100,000 / 400,000 targets of
// up to 2399 rows without / with it: 8 lanes, C = 9 336 / 1303 and 334 / 1305, 11 514 / 1560 and 441 / 1522,
// 13 484 / 1711 and 455 / 1682, 18 634 / 2119 and 547 / 2152, 22 648 / 2531 and 637 / 2491, 26 751 /
// 2944 and 746 / 2958, 28 836 / 3148 and 788 / 3116, 32 891 / 3518 and 893 / 3548; 16 lanes, C = 9 690 /
// 2599 and 655 / 2595, 19 1239 / 4709 and 1196 / 4758, 28 1710 / 6299 and 1545 / 6143, 32 1759 / 7001 and
// 1792 / 7147; 32 lanes, C = 28 3378 / 13490 and 3190 / 12742.
template <int C, bool SEG>
__host__ __device__ constexpr int group_blocks() { return !SEG && (C < 24 || C == 28) ? 1 : 0; }

template <int C, int G, int CI, bool SEG>
__global__ void __launch_bounds__(256, group_blocks<C, SEG>())
msv_ssv_group_kernel(ProfDev P, DbDev db, uint8_t *__restrict__ out_xj, uint8_t *__restrict__ out_flags,
                     unsigned long long *__restrict__ ticket, int64_t *__restrict__ undecided,
                     unsigned long long *__restrict__ n_undecided, int64_t s_begin,
                     const __grid_constant__ SegDev segs) {
  extern __shared__ __align__(16) uint32_t smem[];
  {
    const uint4 *gs = reinterpret_cast<const uint4 *>(P.stab);
    uint4 *ss = reinterpret_cast<uint4 *>(smem);
    for (int i = threadIdx.x; i < group_table_words<C, G, CI>() / 4; i += blockDim.x) ss[i] = __ldg(gs + i);
  }
  __syncthreads();
  const unsigned long long n = SEG ? (unsigned long long) (db.n - segs.nl) + segs.base[segs.S] : (unsigned long long) db.n;
  ssv_group_loop<C, G, CI, SEG>(
      P, smem, db, out_xj, out_flags,
      [&]() -> long long {
        const unsigned long long t = atomicAdd(ticket, 1ull) + (unsigned long long) s_begin;
        return t < n ? (long long) t : -1ll;
      },
      [&](int64_t s) { undecided[atomicAdd(n_undecided, 1ull)] = s; }, segs);
}

// SSV pass of one CTA over the sorted sequences [s0, s0 + nseq) (a work item
// of the multi-profile kernels): next_seq and n_und are shared counters the
// caller zeroed; und (room for nseq entries) receives the chunk-relative
// indices of the undecided sequences. CI > 0: the mixed-width table.
template <int C, int G, int CI = 0>
__device__ __forceinline__ void ssv_group_chunk(const ProfDev &P, const uint32_t *tab, const DbDev &db, int64_t s0,
                                                int nseq, uint8_t *oxj, uint8_t *ofl, unsigned *next_seq,
                                                uint16_t *und, unsigned *n_und) {
  ssv_group_loop<C, G, CI>(
      P, tab, db, oxj, ofl,
      [&]() -> long long {
        const unsigned k = atomicAdd(next_seq, 1u);
        return k < (unsigned) nseq ? (long long) (s0 + k) : -1ll;
      },
      [&](int64_t s) { und[atomicAdd(n_und, 1u)] = (uint16_t) (s - s0); });
}

#ifdef MSVGB_LAUNCHERS_ELSEWHERE
template <int C, int G, int CI = 0> cudaError_t launch_ssv_group(const GroupArgs &a, int num_sms);
#else
template <int C, int G, int CI = 0>
cudaError_t launch_ssv_group(const GroupArgs &a, int num_sms) {
  // without segments the pass has a kernel of its own: their state takes
  // registers (64 -> 78 at 26 words per lane: 3 blocks per SM for 4; 400,000
  // targets in one kernel for both: 3 to 5% longer at most widths below 20
  // words); tables set by hand run without segments
  constexpr bool cuts = CI == hyb_words(C, G);
  if (!cuts && a.segs.S) return cudaErrorInvalidValue;
  auto kern = msv_ssv_group_kernel<C, G, CI, false>;
  if constexpr (cuts) {
    if (a.segs.S) kern = msv_ssv_group_kernel<C, G, CI, true>;
  }
  static_assert(group_words(C, G, CI) == group_table_words<C, G, CI>(), "host and device table sizes agree");
  constexpr size_t smem = (size_t) group_table_words<C, G, CI>() * 4;
  static std::atomic<unsigned long long> configured[2];
  {
    cudaError_t e = ensure_smem_attr((const void *) kern, smem, configured[a.segs.S != 0]);
    if (e != cudaSuccess) return e;
  }
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem);
  if (e != cudaSuccess) return e;
  int grid = std::max(1, per_sm) * num_sms;
  const long long items = a.db.n - a.s_begin - a.segs.nl + (a.segs.S ? a.segs.base[a.segs.S] : 0);
  const long long need = (items * G + 255) / 256;                  // 256 threads hold 256/G sequences
  if (need < grid) grid = (int) std::max(1LL, need);
  (void) cudaGetLastError();
  kern<<<grid, 256, smem, a.stream>>>(a.P, a.db, a.out_xj, a.out_flags, a.ticket, a.undecided, a.n_undecided,
                                      a.s_begin, a.segs);
  return cudaGetLastError();
}
#endif

}  // namespace msvgb

#define MSVGB_INSTANTIATE_GROUP(C, G) \
  template cudaError_t msvgb::launch_ssv_group<C, G, 0>(const msvgb::GroupArgs &, int);
#define MSVGB_INSTANTIATE_HYB(C, G, CI) \
  template cudaError_t msvgb::launch_ssv_group<C, G, CI>(const msvgb::GroupArgs &, int);

namespace msvgb {

// ---- Full MSV (phase B) on lane groups -----------------------------------------
// The sequences SSV leaves undecided are scored with the full MSV recurrence
// (msvfilter.c:112-212) by the same lane groups, 32/G sequences per warp in
// lockstep, instead of one warp per sequence: a lane holds C words (2C cells)
// of its sequence's row, so the per-row work (shuffle, residue decode, the
// row maximum and the J/B updates) is spread over more cells.
//
// Cells are f16 in unit 1, exact: every value is an integer in [0, 255] and
// every sum below 255 + bias. The table (GroupLayout<C, G>, "MSV group
// table") holds c = bias - rbv unclamped, and bias - 255 for padding nodes and
// the pad residue, which keeps those cells at 0 (the previous row's overflow
// test bounds every cell below 255 - bias). Per cell, as msv_row does in
// 16-bit lanes: sv = max(max(mpv, xBc) + c, 0) with xBc = min(xB, 255 - bias).
template <int C, int G>
__device__ __forceinline__ uint32_t msv_row_group(uint32_t (&dp)[C], uint32_t xB2, const uint32_t *__restrict__ tab,
                                                  int x, int glane, int gidx, int src_lane) {
  using Lay = GroupLayout<C, G>;
  using Cp = GroupCopies<G>;
  constexpr uint32_t one2 = 0x3C003C00u;
  uint32_t s[C];
#pragma unroll
  for (int q = 0; q < Lay::Q4; ++q) {
    const uint4 v = *reinterpret_cast<const uint4 *>(tab + (((x * Lay::Q4 + q) * Cp::QUAD + gidx % Cp::QUAD) * G + glane) * 4);
    s[4 * q] = v.x; s[4 * q + 1] = v.y; s[4 * q + 2] = v.z; s[4 * q + 3] = v.w;
  }
  if constexpr (Lay::R >= 2) {
    const int cp = gidx % Cp::PAIR;
    const uint2 v = *reinterpret_cast<const uint2 *>(tab + Lay::A_WORDS + ((x * Cp::PAIR + cp) * G + glane) * 2);
    s[4 * Lay::Q4] = v.x; s[4 * Lay::Q4 + 1] = v.y;
  }
  if constexpr (Lay::R & 1) s[C - 1] = tab[Lay::A_WORDS + Lay::B_WORDS + (x * Cp::SINGLE + gidx) * G + glane];
  const uint32_t pred0 = pred_word0(dp[C - 1], src_lane);
#pragma unroll
  for (int w = C - 1; w >= 0; --w) dp[w] = fma_relu_f16x2(max_f16x2(w ? dp[w - 1] : pred0, xB2), one2, s[w]);
  // the row maximum on the bits (non-negative f16 bits order like integers):
  // one three-input maximum per two words, in four short chains (the
  // maximum is on the critical path of the next row)
  uint32_t acc[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int w = 0; w + 1 < C; w += 2) acc[(w / 2) & 3] = __vimax3_s16x2(acc[(w / 2) & 3], dp[w], dp[w + 1]);
  if constexpr (C & 1) acc[3] = max_s16x2(acc[3], dp[C - 1]);
  return max_s16x2(max_s16x2(acc[0], acc[1]), max_s16x2(acc[2], acc[3]));
}

// Full MSV of the listed sequences list[*ticket .. *list_count) (taken one
// per group from the ticket), written with the full-MSV flag.
// SEG: the longest sequences have been cut, and rows no score depends on are
// skipped. A kernel of its own: the skipping costs every row's chain up to a
// third, and without it a bound of one block per SM makes the chain shorter (us
// for 40 / 2,500 listed targets in the kernel for both and without: 8 lanes, C = 9 491 /
// 496 and 395 / 435, 19 606 / 613 and 440 / 513, 26 573 / 654 and 471 / 566; 16 lanes, C = 10 554 /
// 631 and 444 / 515, 25 671 / 738 and 614 / 719; 32 lanes, C = 24 696 / 831 and 651 / 761).
template <int C, int G, bool SEG>
__global__ void __launch_bounds__(256, SEG ? 0 : 1)
msv_list_group_kernel(ProfDev P, DbDev db, uint8_t *__restrict__ out_xj, uint8_t *__restrict__ out_flags,
                      unsigned long long *__restrict__ ticket, const int64_t *__restrict__ list,
                      const unsigned long long *__restrict__ list_count, const __grid_constant__ SegDev segs) {
  extern __shared__ __align__(16) uint32_t smem[];
  {
    const uint4 *gs = reinterpret_cast<const uint4 *>(P.mtab);
    uint4 *ss = reinterpret_cast<uint4 *>(smem);
    for (int i = threadIdx.x; i < GroupLayout<C, G>::WORDS / 4; i += blockDim.x) ss[i] = __ldg(gs + i);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, glane = lane % G, gbase = lane - glane, gidx = lane / G;
  const int src_lane = gbase + (glane + G - 1) % G;
  const unsigned gmask = (G == 32) ? FULL : (((1u << G) - 1u) << gbase);
  const int tbm = P.tbm, tec = P.tec, base = P.base, bias = P.bias;
  const unsigned long long cnt = *list_count;

  int64_t s = 0;
  int L = 0, i = 0, tjbm = 0, xJ = 0, xB = 0;
  const uint32_t *sq = nullptr;
  uint32_t nextw = kPadWord;
  bool need = true, done = false, er = false;
  int next_blk = -1;                                  // block to look at when its first row comes up
  uint32_t dp[C];
#pragma unroll
  for (int w = 0; w < C; ++w) dp[w] = 0u;

  for (;;) {
    if (need && !done) {                              // group-uniform: take the next listed sequence
      long long t = -1;
      if (glane == 0) {
        const unsigned long long k = atomicAdd(ticket, 1ull);
        if (k < cnt) t = list[k];
      }
      t = __shfl_sync(gmask, t, gbase);
      if (t < 0) {
        done = true;
      } else {
        s = (int64_t) t;
        L = db.len[s];
        tjbm = (P.tjb[L] + tbm) & 0xFF;               // (int8_t) tjb + (int8_t) tbm, splatted as bytes
        xJ = 0;
        xB = max(base - tjbm, 0);
        er = false;
        if constexpr (SEG) next_blk = s < segs.nl ? 0 : -1;
        sq = reinterpret_cast<const uint32_t *>(db.codes + db.start[s]);
        nextw = __ldg(sq);
        i = 0;
        need = false;
#pragma unroll
        for (int w = 0; w < C; ++w) dp[w] = 0u;
      }
    }
    if (__all_sync(FULL, done)) break;
    const bool active = !need && !done;
    if (SEG && active && next_blk >= 0 && i == next_blk * segs.R) {   // rows no score depends on are skipped
      const int nb = (L + segs.R - 1) / segs.R;
      const int k = seg_next_hot(segs, s, nb, next_blk, min(xB, 255 - bias), tec, base, bias, xJ);
      const int r = k * segs.R - segs.warm;
      if (k >= nb) {
        i = L;                                        // no rows left: the sequence ends with this step
      } else if (r > i) {
        i = r;
        nextw = __ldg(sq + (i >> 2));
#pragma unroll
        for (int w = 0; w < C; ++w) dp[w] = 0u;
      }
      next_blk = k + 1;
    }
    const uint32_t w4 = active ? nextw : kPadWord;
    if (active && i + 4 < L) nextw = __ldg(sq + (i >> 2) + 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t xb = (uint32_t) __half_as_ushort(__int2half_rn(min(xB, 255 - bias)));
      uint32_t a = msv_row_group<C, G>(dp, xb | (xb << 16), smem, (w4 >> (8 * j)) & 0xFF, glane, gidx, src_lane);
      int m = max((int) (a & 0xFFFFu), (int) (a >> 16));   // f16 bits of values in [0, 255]
#pragma unroll
      for (int off = G / 2; off >= 1; off >>= 1) m = max(m, __shfl_xor_sync(FULL, m, off));
      const int xE = (int) __half2float(__ushort_as_half((unsigned short) m));
      if (active && !er && i + j < L) {               // rows past the end change nothing
        if (xE + bias >= 255) er = true;              // adds(xE, bias) == 255: +inf
        else {
          xJ = max(xJ, max(xE - tec, 0));
          xB = max(max(base, xJ) - tjbm, 0);
        }
      }
    }
    i += 4;
    if (active && (er || i >= L)) {
      if (glane == 0) {
        const int64_t oi = db.orig[s];
        int flags = 0x04;
        if (er) flags |= 0x01 | 0x02;
        else if (xJ >= P.xjmin[L]) flags |= 0x02;
        out_xj[oi] = (uint8_t) (er ? 255 : xJ);
        out_flags[oi] = (uint8_t) flags;
      }
      need = true;
    }
  }
}

#ifdef MSVGB_LAUNCHERS_ELSEWHERE
template <int C, int G>
cudaError_t launch_list_group(const ProfDev &P, const DbDev &db, uint8_t *out_xj, uint8_t *out_flags,
                              unsigned long long *ticket, const int64_t *list, const unsigned long long *list_count,
                              const SegDev &segs, int num_sms, cudaStream_t stream);
#else
template <int C, int G>
cudaError_t launch_list_group(const ProfDev &P, const DbDev &db, uint8_t *out_xj, uint8_t *out_flags,
                              unsigned long long *ticket, const int64_t *list, const unsigned long long *list_count,
                              const SegDev &segs, int num_sms, cudaStream_t stream) {
  auto kern = segs.S ? msv_list_group_kernel<C, G, true> : msv_list_group_kernel<C, G, false>;
  constexpr size_t smem = (size_t) GroupLayout<C, G>::WORDS * 4;
  static std::atomic<unsigned long long> configured[2];
  {
    cudaError_t e = ensure_smem_attr((const void *) kern, smem, configured[segs.S != 0]);
    if (e != cudaSuccess) return e;
  }
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem);
  if (e != cudaSuccess) return e;
  // a block per SM holds a small search's list (about a 16th of the sequences
  // at most, as a rule) and leaves the rest of the SM to searches on other
  // streams; larger lists fill the SMs
  constexpr int groups = 256 / G;
  const long long want = (db.n / 16 + groups - 1) / groups;
  const long long grid = std::max<long long>(num_sms, std::min<long long>((long long) std::max(1, per_sm) * num_sms, want));
  (void) cudaGetLastError();
  kern<<<(unsigned) grid, 256, smem, stream>>>(P, db, out_xj, out_flags, ticket, list, list_count, segs);
  return cudaGetLastError();
}
#endif

}  // namespace msvgb

#define MSVGB_INSTANTIATE_LIST(C, G)                                                                       \
  template cudaError_t msvgb::launch_list_group<C, G>(const msvgb::ProfDev &, const msvgb::DbDev &, uint8_t *, \
                                                      uint8_t *, unsigned long long *, const int64_t *,      \
                                                      const unsigned long long *, const msvgb::SegDev &, int, \
                                                      cudaStream_t);
