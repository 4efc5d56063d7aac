// msv_kernel_impl.cuh -- the search kernel and its launcher (instantiated per C
// in inst_*.cu so the translation units compile in parallel).
#pragma once
#include <cuda_fp16.h>
#include "msv_device.cuh"

namespace msvgb {

struct LaunchArgs {
  ProfDev             P;
  DbDev               db;
  uint8_t            *out_xj;     // [n] in original sequence order
  uint8_t            *out_flags;  // [n]
  unsigned long long *ticket;     // zeroed before the launch
  cudaStream_t        stream;
  int                 grid;       // 0: fill the GPU
  int                 skip_empty; // 1: L == 0 is skipped as p7_Pipeline does; 0: scored like p7_MSVFilter
  // Range mode (range_end > 0): only the sorted sequences [0, range_end).
  int64_t                   range_end = 0;
  // Segments of the longest sequences (not in range mode).
  SegDev                    segs{};
};

constexpr int WARPS_PER_CTA = 8;
constexpr int MAX_WARPS_PER_CTA = 16;   // used when the tables leave room for one CTA per SM

// f16 tables wider than 40 words per lane (M >= 2560: 154 KB of SSV costs
// and up) do not fit in shared memory beside the MSV table: such profiles keep
// both tables in global memory, where they stream through L1 and L2 (a few
// hundred KB, resident in the 129 MB L2 for the whole launch).
template <int C, bool F16>
__host__ __device__ constexpr bool tables_in_global() { return F16 && C > 40; }

template <int C, bool F16>
constexpr size_t smem_bytes() {   // SSV table + MSV table
  if (tables_in_global<C, F16>()) return 0;
  return ((size_t) (F16 ? NRES * C * 32 : NRES * (C / 2) * 32) + (size_t) NRES * ((C + 1) / 2) * 32) * 4;
}

// Threads per CTA: 8 warps, or 16 when the tables leave room for only one CTA per SM.
template <int C, bool F16>
constexpr int cta_threads() { return 2 * smem_bytes<C, F16>() > 227 * 1024 ? MAX_WARPS_PER_CTA * 32 : WARPS_PER_CTA * 32; }

// Words of four residues per step of the SSV loop. Narrow rows go eight a step,
// so that the next rows' costs are loaded under a row's shuffle (M = 200, 20,000
// targets: 217 us, 251 at four; M = 400, 40,000: 552 and 611; one call of the
// drop-in at M = 200: 29 us and 34); from 9 words four rows keep as much in flight
// (M = 700: 716 and 744, 900: 689 and 672).
template <int C, bool F16>
__host__ __device__ constexpr int row_words() { return F16 && C <= 8 ? 2 : 1; }

// Both tables into shared memory, unless they stay in global memory.
template <int C, bool F16>
__device__ __forceinline__ void stage_tables(uint32_t *smem, const uint32_t *&stab, const uint32_t *&mtab) {
  constexpr int SW = F16 ? NRES * C * 32 : NRES * (C / 2) * 32;   // words of the SSV table
  constexpr int MW = NRES * ((C + 1) / 2) * 32;                    // words of the MSV table
  if constexpr (!tables_in_global<C, F16>()) {
    const uint4 *gs = reinterpret_cast<const uint4 *>(stab);
    const uint4 *gm = reinterpret_cast<const uint4 *>(mtab);
    uint4 *ss = reinterpret_cast<uint4 *>(smem);
    uint4 *sm = reinterpret_cast<uint4 *>(smem + SW);
    for (int i = threadIdx.x; i < SW / 4; i += blockDim.x) ss[i] = __ldg(gs + i);
    for (int i = threadIdx.x; i < MW / 4; i += blockDim.x) sm[i] = __ldg(gm + i);
    stab = smem;
    mtab = smem + SW;
    __syncthreads();
  }
}

// Persistent kernel for searches that cut their long targets (segs.S > 0;
// msv_whole_kernel otherwise): every CTA stages the profile's cost tables into
// shared memory once, then its warps pull segments and whole sequences
// (longest first) from a global ticket until the database is exhausted. Bound by
// shared memory where the database fills the SMs (2 bytes of cost per cell),
// by the longest chain of rows where it does not (SegDev).
template <int C, bool F16>
__global__ void __launch_bounds__(cta_threads<C, F16>())
msv_search_kernel(ProfDev P, DbDev db, uint8_t *__restrict__ out_xj, uint8_t *__restrict__ out_flags,
                  unsigned long long *__restrict__ ticket, int skip_empty,
                  int64_t range_end, const __grid_constant__ SegDev segs) {
  extern __shared__ __align__(16) uint32_t smem[];
  const uint32_t *stab = P.stab, *mtab = P.mtab;
  stage_tables<C, F16>(smem, stab, mtab);
  const int lane = threadIdx.x & 31;
  const unsigned long long nseg = segs.S ? segs.base[segs.S] : 0ull;
  const unsigned long long nitems = (unsigned long long) (range_end > 0 ? range_end : db.n - segs.nl) + nseg;
  for (;;) {
    unsigned long long s = 0;
    if (lane == 0) s = atomicAdd(ticket, 1ull);
    s = __shfl_sync(FULL, s, 0);
    if (s >= nitems) break;
    const unsigned long long item = s;
    int k = -1;                                       // segment index
    if (item < nseg) { k = seg_of(segs, (uint32_t) item); s = item - segs.base[k]; }
    else s = item - nseg + (unsigned long long) segs.nl;
    const int L = db.len[s];
    const int64_t oi = db.orig[s];
    if (L == 0 && skip_empty) {
      if (lane == 0) { out_xj[oi] = 0; out_flags[oi] = 0x08; }   // MSVGB_FLAG_EMPTY
      continue;
    }
    const uint32_t *sq = reinterpret_cast<const uint32_t *>(db.codes + db.start[s]);
    const int tjb = P.tjb[L];
    const bool ssv_off = tjb + P.tbm + P.tec + P.bias >= 127;   // SSV disabled for this length
    int xj, full = 0, st = -1;
    if (k >= 0 || !ssv_off) {
      const int r0 = k >= 0 ? k * segs.T : 0, end = k >= 0 ? min(L, r0 + segs.T) : L;
      int umax = ssv_range<C, F16, row_words<C, F16>()>(stab, sq, max(0, r0 - segs.warm), end, lane, k >= 0 ? &segs : nullptr,
                                   (int64_t) s, r0);
      if (k >= 0) {                                   // the sequence's last segment to finish decides it
        if (lane == 0) umax = seg_finish(segs, (int64_t) s, L);
        __syncwarp();                                 // the other lanes read u[] too (msv_full): behind lane 0's fence
        umax = __shfl_sync(FULL, umax, 0);
        if (umax < 0) continue;
      }
      if (!ssv_off) st = ssv_decide(umax, tjb, P.tbm, P.tec, P.base, P.bias, xj);
    }
    if (st < 0) {
      full = 1;
      st = msv_full<C>(P, mtab, sq, L, tjb, lane, xj, k >= 0 ? &segs : nullptr, (int64_t) s);
    }
    if (lane == 0) {
      int flags = full ? 0x04 : 0;
      if (st == ST_ERANGE) flags |= 0x01 | 0x02;                 // +inf always passes F1
      else if (xj >= P.xjmin[L]) flags |= 0x02;
      out_xj[oi] = (uint8_t) xj;
      out_flags[oi] = (uint8_t) flags;
    }
  }
}

// Blocks per SM that the whole-sequence kernel is compiled for (0: the
// compiler's own choice), and words of four residues per step of its SSV loop.
template <int C, bool F16>
__host__ __device__ constexpr int whole_blocks() { return !F16 || C <= 32 ? 1 : 0; }
template <int C, bool F16>
__host__ __device__ constexpr int whole_words() { return F16 && C > 8 && C <= 32 ? 1 : 2; }

// The same search with no sequence cut: long targets beside a lane-group pass,
// chunks of a host search, calls that may not allocate. A warp's time is then
// the chain of the longest rows it scores, and how far ahead of it the
// compiler loads the costs sets that chain: a bound of one block per SM frees
// the registers for it, eight rows a step give it room (from 9 to 32 words they
// shorten the SSV row but lengthen the full MSV's: M = 760, 60,000 targets 1659 us
// with eight, 1566 with four). ns per row of one warp, SSV / full MSV, in the
// kernel for both and here (f16 tables): C = 1 23.4 / 143 and 21.5 / 129, 3 35.0 / 151
// and 18.0 / 135, 6 45.4 / 163 and 18.4 / 144, 11 47.0 / 175 and 33.5 / 156, 16 47.1 / 199 and
// 37.8 / 173, 21 52.5 / 194 and 45.0 / 178, 32 71.0 / 261 and 67.2 / 233, 52 129 / 396 and
// 103 / 395 (with the bound 101 / 404), 96 292 / 1090 and 270 / 1029 (with it 368 for the SSV
// row, and 34% longer where the SMs are full).
template <int C, bool F16>
__global__ void __launch_bounds__(cta_threads<C, F16>(), whole_blocks<C, F16>())
msv_whole_kernel(ProfDev P, DbDev db, uint8_t *__restrict__ out_xj, uint8_t *__restrict__ out_flags,
                 unsigned long long *__restrict__ ticket, int skip_empty, int64_t range_end) {
  extern __shared__ __align__(16) uint32_t smem[];
  const uint32_t *stab = P.stab, *mtab = P.mtab;
  stage_tables<C, F16>(smem, stab, mtab);
  const int lane = threadIdx.x & 31;
  const unsigned long long nitems = (unsigned long long) (range_end > 0 ? range_end : db.n);
  for (;;) {
    unsigned long long s = 0;
    if (lane == 0) s = atomicAdd(ticket, 1ull);
    s = __shfl_sync(FULL, s, 0);
    if (s >= nitems) break;
    const int L = db.len[s];
    const int64_t oi = db.orig[s];
    if (L == 0 && skip_empty) {
      if (lane == 0) { out_xj[oi] = 0; out_flags[oi] = 0x08; }   // MSVGB_FLAG_EMPTY
      continue;
    }
    const uint32_t *sq = reinterpret_cast<const uint32_t *>(db.codes + db.start[s]);
    int xj, full;
    const int st = msv_one<C, F16, whole_words<C, F16>()>(P, stab, mtab, sq, L, lane, xj, full);
    if (lane == 0) {
      int flags = full ? 0x04 : 0;
      if (st == ST_ERANGE) flags |= 0x01 | 0x02;                 // +inf always passes F1
      else if (xj >= P.xjmin[L]) flags |= 0x02;
      out_xj[oi] = (uint8_t) xj;
      out_flags[oi] = (uint8_t) flags;
    }
  }
}

#ifdef MSVGB_LAUNCHERS_ELSEWHERE
template <int C, bool F16> cudaError_t launch_search(const LaunchArgs &a, int num_sms);
#else
template <int C, bool F16>
cudaError_t launch_search(const LaunchArgs &a, int num_sms) {
  const bool cut = a.segs.S != 0;
  const void *kern = cut ? (const void *) msv_search_kernel<C, F16> : (const void *) msv_whole_kernel<C, F16>;
  constexpr size_t smem = smem_bytes<C, F16>();
  static std::atomic<unsigned long long> configured[2];
  {
    cudaError_t e = ensure_smem_attr(kern, smem, configured[cut]);
    if (e != cudaSuccess) return e;
  }
  constexpr int threads = cta_threads<C, F16>();
  int grid = a.grid;
  if (grid <= 0) {
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    // Where long targets are cut the chains set the time, and they run faster
    // with fewer warps beside them (8 / 4 / 3 / 2 blocks per SM, us: M = 130, 40,000
    // targets 369 / 370 / 381 / 431; M = 400, 5,000 261 / 260 / 248 / 232, 40,000 552 / 553 / 484 /
    // 483; M = 550, 10,000 334 / 329 / 310 / 286, 60,000 872 / 876 / 834 / 844; M = 800, 10,000 393 /
    // 392 / 398 / 344; 4 / 3 blocks at M = 225: 5,000 189 / 173, 20,000 241 / 233, 40,000 348 / 335).
    if (F16 && cut) per_sm = std::min(per_sm, C <= 3 ? 4 : C == 4 ? 3 : 2);
    grid = per_sm * num_sms;
    const int warps = threads / 32;
    const long long items = a.range_end > 0 ? a.range_end : a.db.n - a.segs.nl + (a.segs.S ? a.segs.base[a.segs.S] : 0);
    const long long need = (items + warps - 1) / warps;
    if (need < grid) grid = (int) (need > 0 ? need : 1);
  }
  (void) cudaGetLastError();   // clear a stale error left by an unrelated call
  if (cut)
    msv_search_kernel<C, F16><<<grid, threads, smem, a.stream>>>(a.P, a.db, a.out_xj, a.out_flags, a.ticket, a.skip_empty,
                                                                 a.range_end, a.segs);
  else
    msv_whole_kernel<C, F16><<<grid, threads, smem, a.stream>>>(a.P, a.db, a.out_xj, a.out_flags, a.ticket, a.skip_empty,
                                                                a.range_end);
  return cudaGetLastError();
}
#endif

}  // namespace msvgb

#define MSVGB_INSTANTIATE_I8(C) \
  template cudaError_t msvgb::launch_search<C, false>(const msvgb::LaunchArgs &, int);
#define MSVGB_INSTANTIATE_F16(C) \
  template cudaError_t msvgb::launch_search<C, true>(const msvgb::LaunchArgs &, int);
