// msv_bias.cu -- the bias filter of p7_Pipeline on the GPU, and the gate of
// every filter stage.
//
// p7_bg_FilterScore (src/p7_bg.c:473-483) scores a sequence with a two-state
// HMM: state 0 emits the background composition, state 1 the model's
// (p7_bg_SetFilter, src/p7_bg.c:431-453, with p7_bg_SetLength's t[0][0]);
// esl_hmm_Forward (easel/esl_hmm.c:351-409) runs it scaled, dividing every
// row by its maximum and summing the logs of those maxima. The recurrence is
// sequential in the residues and has two states, so a few lanes score one
// listed sequence, with the reference's float operations in its order:
// round-to-nearest multiplies, adds and divides written as intrinsics (no
// contraction into FMA), and each row's log taken in double and rounded to
// float as the reference's double log() of a float is. The double log is a
// table-driven one (Tang's method, ACM TOMS 15(2), 1989: reduce by a table
// entry, then a short polynomial; here 512 entries and the Taylor series of
// log1p to degree 6), about 8 double operations instead of the library
// log's many more on this part's narrow FP64 pipe; a row whose result lies
// within 64 units in the last place of a float rounding boundary takes the
// library log instead. The length term (logf of p1 and 1 - p1) is added on the host with
// the C library's logf.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/msvgb.h"
#include "msv_internal.h"

using namespace msvgb;
using msvgb_detail::fail;

namespace {

constexpr int kLogTab = 512;

struct BiasDev {
  float eo[NRES][2];       // emission odds: [x][0] background state, [x][1] model-composition state
  float t10, t11;          // biased-state transitions 1->0, 1->1 (t[1][2] = 1)
  float pi0, pi1;
  double2 logtab[kLogTab]; // per top-9-mantissa-bit interval: (1/c, log c) of its reduction point c
};

// float(log((double) m)) for a float m > 0: m = 2^e f, f in [1, 2); the top 9
// bits of f pick the interval [1 + j/512, 1 + (j+1)/512), whose point c is its
// midpoint (halved, with e + 1, from j = 212 (f > 1.414) up, so that f/c stays
// near 1 and no sum cancels); the intervals next to 1 use c = 1 (m near 1:
// log m = log1p(f - 1), no table term). f, halved or not, is assembled as a
// double from the float's bits. log m = e ln2 + log c + log1p(r), r = f (1/c)
// - 1 by one fused multiply-add, |r| < 2^-9; log1p to degree 6 (truncation <
// 2^-56 relative). The result's distance to the nearest float rounding
// boundary is read from the low 29 bits of the double: within 64 units of the
// last place the library log decides instead.
__device__ __forceinline__ float log_row(float m, const double2 *tab) {
  const uint32_t b = __float_as_uint(m);
  if (b - 0x00800000u >= 0x7f000000u) return (float) log((double) m);   // 0, subnormal, inf, nan, negative
  const int j = (b >> 14) & 0x1ff;
  const int half = j >= 212;
  const int e = (int) (b >> 23) - 127 + half;
  const double f = __longlong_as_double((long long) (((uint64_t) (b & 0x7fffffu) << 29) |
                                                     ((uint64_t) (1023 - half) << 52)));
  const double2 t = tab[j];
  const double r = fma(f, t.x, -1.0);
  double p = fma(-1.0 / 6, r, 1.0 / 5);
  p = fma(p, r, -1.0 / 4);
  p = fma(p, r, 1.0 / 3);
  p = fma(p, r, -1.0 / 2);
  p = fma(p, r, 1.0);
  double y;
  if (e == 0) {
    y = fma(p, r, t.y);
  } else {
    const double ln2_hi = 6.93147180369123816490e-01, ln2_lo = 1.90821492927058770002e-10;
    const double de = (double) e;
    y = fma(de, ln2_hi, t.y + fma(de, ln2_lo, p * r));
  }
  const long long dist = (long long) ((uint64_t) __double_as_longlong(y) & 0x1fffffffull) - 0x10000000ll;
  if (dist > -64 && dist < 64) return (float) log((double) m);      // near a float rounding boundary
  return __double2float_rn(y);
}

// float(log(m)) in float-float arithmetic on the FP32 pipe, for m in
// [2^-8.5, 2^8.5) (exponents -8 .. 8 after the reduction; the row maxima of
// the filter's scaled Forward lie there): the top 11 mantissa bits pick a
// reduction point c (2048 intervals; c = 1 next to 1) with 1/c and log c
// stored as float pairs; d = f - c is exact, r = d/c a float pair by fused
// multiply-adds, log1p(r) = r - r^2/2 (pairs) + r^3/3 - r^4/4 + r^5/5 (float;
// |r| < 2^-11.5, truncation < 2^-57), summed with error-free two-sums. The
// result is returned only when it is at least 2^-42 (relative) away from a
// float rounding boundary -- every float in [2^-8, 2^8) checked on the host
// against the C library's double log: 0 differences, 737 of 134 M left to
// the double path; otherwise (and for other exponents) the double path
// decides.
__device__ float4 g_logff[2048];

__device__ __forceinline__ float fsub(float a, float b) { return __fadd_rn(a, -b); }

// Branch-free: ok says whether the returned value is the result (the
// arithmetic runs on any input; the table index is always in range).
__device__ __forceinline__ float log_ff(float m, bool &ok) {
  const uint32_t b = __float_as_uint(m);
  const int j = (b >> 12) & 0x7ff;
  const int half = j >= 849;
  const int e = (int) (b >> 23) - 127 + half;
  const bool in_range = b - 0x00800000u < 0x7f000000u && e >= -8 && e <= 8;
  const float f = __uint_as_float((b & 0x7fffffu) | ((uint32_t) (127 - half) << 23));
  const float4 t = g_logff[j];                               // 1/c (hi, lo), log c (hi, lo)
  const float c = (j == 0 || j == 2047) ? 1.0f : __fmul_rn(half ? 0.5f : 1.0f, 1.0f + ((float) j + 0.5f) / 2048.0f);
  const float d = fsub(f, c);                                // exact
  const float rh = __fmul_rn(d, t.x);
  const float rl = __fadd_rn(__fmaf_rn(d, t.x, -rh), __fmul_rn(d, t.y));
  const float sh = __fmul_rn(rh, rh);
  const float sl = __fadd_rn(__fmaf_rn(rh, rh, -sh), __fmul_rn(__fmul_rn(2.0f, rh), rl));
  const float q3 = __fmul_rn(__fmul_rn(rh, sh),
                             __fadd_rn(1.0f / 3.0f, __fmul_rn(rh, __fadd_rn(-0.25f, __fmul_rn(rh, 0.2f)))));
  // e ln2 in three parts: a 16-bit head (e * head exact for |e| <= 8), the
  // middle as an exact product, the tail
  const float l2h = 0.693145751953125f, l2m = 0x1.7f7d1cp-20f, l2l = 5.49560397e-14f;
  const float fe = (float) e;
  const float A = __fmul_rn(fe, l2h);
  const float bh = __fmul_rn(fe, l2m), bl = __fmaf_rn(fe, l2m, -bh);
  float H = A, L = 0.0f, sm, bb;
  auto two_sum = [&](float x) {                              // H + x = sm + error, the error into L
    sm = __fadd_rn(H, x); bb = fsub(sm, H);
    L = __fadd_rn(L, __fadd_rn(fsub(H, fsub(sm, bb)), fsub(x, bb)));
    H = sm;
  };
  two_sum(t.z);
  two_sum(bh);
  two_sum(rh);
  two_sum(__fmul_rn(-0.5f, sh));
  L = __fadd_rn(L, __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(t.w, bl), __fmul_rn(fe, l2l)), rl),
                                       __fmul_rn(-0.5f, sl)), q3));
  const float res = __fadd_rn(H, L);
  const float bv = fsub(res, H);
  const float tr = __fadd_rn(fsub(H, fsub(res, bv)), fsub(L, bv));   // H + L - res, exactly
  const uint32_t rb = __float_as_uint(res);
  const float ulp = __uint_as_float((rb & 0x7f800000u) - (23u << 23));
  ok = in_range && (rb & 0x7fffffffu) >= 0x01000000u &&
       !(fsub(__fmul_rn(0.5f, ulp), fabsf(tr)) < __fmul_rn(fabsf(res), 0x1p-42f));
  return res;
}

__device__ __forceinline__ float log_rowf(float m, const double2 *tab) {
  bool ok;
  const float r = log_ff(m, ok);
  return ok ? r : log_row(m, tab);
}

// G lanes per listed sequence (groups take the list in database order, the
// longest first, so a warp's sequences have similar lengths). Every lane of a
// group runs the recurrence -- the serial chain through the divisions, which
// is what a sequence's time consists of -- and the row logs, which are off the
// chain, are split over the lanes: rows go 16 at a time, lane g taking the
// logs of rows g, g + G, ... of one batch while the next batch's recurrence
// runs, and their sum is taken in row order through shuffles. (With one thread
// per sequence a warp issued 150 instructions per row of one chain: 1.97 ms
// for a call on 40,000 listed sequences, 1.08 so.)
//
// ONE: the row's larger value divided by itself is 1, so only the smaller one
// is divided; the host checks that the filter's odds and transitions keep the
// maximum positive and finite in every row (else both are divided, as the
// reference does).
template <bool ONE>
__device__ __forceinline__ float bias_scale(float n0, float n1, float &d0, float &d1) {
  if constexpr (ONE) {
    const bool first = n0 >= n1;
    const float m = first ? n0 : n1, r = __fdiv_rn(first ? n1 : n0, m);
    d0 = first ? 1.0f : r;
    d1 = first ? r : 1.0f;
    return m;
  } else {
    float m = 0.0f;                              // ESL_MAX(dp, max) over k = 0, 1
    m = n0 > m ? n0 : m;
    m = n1 > m ? n1 : m;
    d0 = __fdiv_rn(n0, m);
    d1 = __fdiv_rn(n1, m);
    return m;
  }
}

// Rows of one batch: the row maxima of this lane's rows into nm; rows at or
// past live (FULL: none) are dropped. FIRST: the first row starts from pi.
template <int G, bool ONE, bool FIRST, bool FULL>
__device__ __forceinline__ void bias_rows(const BiasDev &B, const float2 *s_eo, const uint4 w, int live, int glane,
                                          float t00, float t01, float &d0, float &d1, float (&nm)[16 / G]) {
  const uint32_t words[4] = {w.x, w.y, w.z, w.w};
  // the odds first: the divisions branch (a rare slow path), and no load
  // would be moved across one into the chain's latency
  float2 eo[16];
#pragma unroll
  for (int b = 0; b < 16; ++b) eo[b] = s_eo[(words[b >> 2] >> (8 * (b & 3))) & 0xff];
#pragma unroll
  for (int b = 0; b < 16; ++b) {
    if (!FULL && b >= live) break;
    const float2 e = eo[b];
    float n0, n1;
    if (FIRST && b == 0) {
      n0 = __fmul_rn(e.x, B.pi0);
      n1 = __fmul_rn(e.y, B.pi1);
    } else {
      n0 = __fmul_rn(__fadd_rn(__fmul_rn(d0, t00), __fmul_rn(d1, B.t10)), e.x);
      n1 = __fmul_rn(__fadd_rn(__fmul_rn(d0, t01), __fmul_rn(d1, B.t11)), e.y);
    }
    const float m = bias_scale<ONE>(n0, n1, d0, d1);
    if (b % G == glane) nm[b / G] = m;
  }
}

// The logs of this lane's maxima; bit k of the result: log k is not decided.
template <int K>
__device__ __forceinline__ uint32_t bias_logs(const float (&mx)[K], float (&lg)[K]) {
  uint32_t fail = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    bool ok;
    lg[k] = log_ff(mx[k], ok);
    fail |= ok ? 0u : 1u << k;
  }
  return fail;
}

// Adds a batch's first n row logs to logsc, in row order.
template <int G>
__device__ __forceinline__ void bias_add(const float (&mx)[16 / G], float (&lg)[16 / G], uint32_t fail, int n,
                                         const double2 *s_log, unsigned gmask, float &logsc) {
  if (fail) {
#pragma unroll
    for (int k = 0; k < 16 / G; ++k)
      if (fail >> k & 1u) lg[k] = log_row(mx[k], s_log);
  }
  __syncwarp(gmask);
#pragma unroll
  for (int b = 0; b < 16; ++b) {
    const float v = __shfl_sync(gmask, lg[b / G], b % G, G);
    logsc = b < n ? __fadd_rn(logsc, v) : logsc;
  }
}

// Shared-memory copies of the filter's odds and the log table.
struct BiasShared {
  float2 eo[NRES];
  double2 logtab[kLogTab];
  __device__ __forceinline__ void load(const BiasDev &B) {
    for (int i = threadIdx.x; i < NRES; i += blockDim.x) eo[i] = make_float2(B.eo[i][0], B.eo[i][1]);
    for (int i = threadIdx.x; i < kLogTab; i += blockDim.x) logtab[i] = B.logtab[i];
    __syncthreads();
  }
};

// The Forward score of one sequence, without its length terms.
template <int G, bool ONE>
__device__ __forceinline__ float bias_score(const BiasDev &B, const BiasShared &sh, const uint4 *sq, int L, int glane,
                                            unsigned gmask) {
  constexpr int K = 16 / G;                      // logs per lane and batch
  const float t00 = __fdiv_rn((float) L, (float) (L + 1)), t01 = __fadd_rn(1.0f, -t00);
  float d0 = 0.0f, d1 = 0.0f, logsc = 0.0f;
  float mx[K], lg[K];                            // this lane's row maxima of the last batch, logs not yet taken
#pragma unroll
  for (int k = 0; k < K; ++k) mx[k] = 1.0f;
  bias_rows<G, ONE, true, false>(B, sh.eo, sq[0], L, glane, t00, t01, d0, d1, mx);
  int i0 = 16;
  for (; i0 + 16 <= L; i0 += 16) {               // the previous batch (rows i0-16 .. i0-1) is full
    float nm[K];
    const uint32_t fail = bias_logs(mx, lg);
    bias_rows<G, ONE, false, true>(B, sh.eo, sq[i0 >> 4], 16, glane, t00, t01, d0, d1, nm);
    bias_add<G>(mx, lg, fail, 16, sh.logtab, gmask, logsc);
#pragma unroll
    for (int k = 0; k < K; ++k) mx[k] = nm[k];
  }
  if (i0 < L) {
    float nm[K];
#pragma unroll
    for (int k = 0; k < K; ++k) nm[k] = 1.0f;
    const uint32_t fail = bias_logs(mx, lg);
    bias_rows<G, ONE, false, false>(B, sh.eo, sq[i0 >> 4], L - i0, glane, t00, t01, d0, d1, nm);
    bias_add<G>(mx, lg, fail, 16, sh.logtab, gmask, logsc);
#pragma unroll
    for (int k = 0; k < K; ++k) mx[k] = nm[k];
  }
  const uint32_t fail = bias_logs(mx, lg);
  bias_add<G>(mx, lg, fail, (L - 1) % 16 + 1, sh.logtab, gmask, logsc);
  return __fadd_rn(logsc, log_rowf(__fadd_rn(d0, d1), sh.logtab));   // dp[L][0] * 1 + dp[L][1] * 1
}

// ---- long sequences in segments ---------------------------------------------------
// The chain of a long sequence is cut into segments of kBiasSeg rows that run
// side by side. A segment does not know the state (d0, d1) it starts from: it
// starts kBiasWarm rows early from a guess. The filter forgets its state (each
// row's map contracts, by t11 and the odds of the two compositions), so after
// the run-in two runs are usually equal in every bit, rounding included; and
// when the state a segment had at its first row equals, bit for bit, the state
// the segment before ended in, its rows are the sequence's own. That is
// checked for every segment, and a sequence that fails is scored from its
// start, so no result depends on the guess. The row logs go to memory and are
// summed in row order by one thread: four clocks a row against about 180 for
// the chain.
//
// Run-in of 1024 rows: in a float simulation on background sequences, runs
// from the guess still differed after 512 rows in 26% of cases with the
// Pkinase model (composition close to the background: it forgets slowest),
// after 768 in 0.05%, and in none of 4,000 with four other models after 512.
constexpr int kBiasSeg = 512, kBiasWarm = 1024, kBiasLong = 3 * kBiasSeg;

struct BiasSegs {                                // of one call; counters zeroed
  unsigned *n;                                   // [0] long sequences, [1] segments, [2] rows
  unsigned cap_seq, cap_item, cap_row;           // rows in units of kBiasSeg
  int32_t *seq;                                  // [cap_seq] list position
  unsigned *first, *row;                         // [cap_seq] first segment, first block of rows in lg
  uint2 *item;                                   // [cap_item] long sequence, segment
  float4 *state;                                 // [cap_item] (d0, d1) before its first row and after its last
  float *lg;                                     // [cap_row * kBiasSeg] row logs
  uint8_t *is_long;                              // [nids]
};

// Picks the long sequences of the list while there is room for them.
__global__ void __launch_bounds__(256)
bias_plan_kernel(DbDev db, const int64_t *__restrict__ slots, int64_t nids, BiasSegs S) {
  const int64_t j = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nids) return;
  const int L = db.len[slots[j]];
  uint8_t is_long = 0;
  if (L > kBiasLong) {
    const unsigned nseg = (unsigned) (L + kBiasSeg - 1) / kBiasSeg;
    const unsigned r = atomicAdd(&S.n[2], nseg);
    if (r + nseg <= S.cap_row) {                 // cap_seq and cap_item are cap_row or more
      const unsigned e = atomicAdd(&S.n[0], 1u), f = atomicAdd(&S.n[1], nseg);
      S.seq[e] = (int32_t) j;
      S.first[e] = f;
      S.row[e] = r;
      for (unsigned k = 0; k < nseg; ++k) S.item[f + k] = make_uint2(e, k);
      is_long = 1;
    }
  }
  S.is_long[j] = is_long;
}

template <int G, bool ONE>
__device__ __forceinline__ void bias_segment(const BiasDev &B, const BiasShared &sh, const DbDev &db,
                                             const int64_t *slots, const BiasSegs &S, unsigned it, int glane) {
  constexpr int K = 16 / G;
  const uint2 item = S.item[it];
  const int64_t s = slots[S.seq[item.x]];
  const int L = db.len[s], r0 = (int) item.y * kBiasSeg, r1 = min(L, r0 + kBiasSeg);
  const uint4 *sq = reinterpret_cast<const uint4 *>(db.codes + db.start[s]);
  float *lg_out = S.lg + (size_t) (S.row[item.x] + item.y) * kBiasSeg;
  const float t00 = __fdiv_rn((float) L, (float) (L + 1)), t01 = __fadd_rn(1.0f, -t00);
  float d0 = 1.0f, d1 = 0.05f;                   // the guess
  float mx[K], nm[K], lg[K];
  int i = r0 == 0 ? 0 : r0 - kBiasWarm;
  if (i <= 0 && r0 > 0) {                        // no guess: from the sequence's start
    bias_rows<G, ONE, true, false>(B, sh.eo, sq[0], 16, glane, t00, t01, d0, d1, nm);
    i = 16;
  }
  for (; i < r0; i += 16)
    bias_rows<G, ONE, false, true>(B, sh.eo, sq[i >> 4], 16, glane, t00, t01, d0, d1, nm);
  const float s0 = d0, s1 = d1;
  // as bias_score: the logs of one batch beside the next batch's recurrence
  auto store = [&](int row, uint32_t fail) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      lg_out[row + k * G + glane] = (fail >> k & 1u) ? log_row(mx[k], sh.logtab) : lg[k];
  };
#pragma unroll
  for (int k = 0; k < K; ++k) mx[k] = 1.0f;
  if (r0 == 0) bias_rows<G, ONE, true, false>(B, sh.eo, sq[0], 16, glane, t00, t01, d0, d1, mx);
  else         bias_rows<G, ONE, false, false>(B, sh.eo, sq[r0 >> 4], r1 - r0, glane, t00, t01, d0, d1, mx);
  int i0 = r0 + 16;
  for (; i0 + 16 <= r1; i0 += 16) {
    const uint32_t fail = bias_logs(mx, lg);
    bias_rows<G, ONE, false, true>(B, sh.eo, sq[i0 >> 4], 16, glane, t00, t01, d0, d1, nm);
    store(i0 - 16 - r0, fail);
#pragma unroll
    for (int k = 0; k < K; ++k) mx[k] = nm[k];
  }
  if (i0 < r1) {
#pragma unroll
    for (int k = 0; k < K; ++k) nm[k] = 1.0f;
    const uint32_t fail = bias_logs(mx, lg);
    bias_rows<G, ONE, false, false>(B, sh.eo, sq[i0 >> 4], r1 - i0, glane, t00, t01, d0, d1, nm);
    store(i0 - 16 - r0, fail);
#pragma unroll
    for (int k = 0; k < K; ++k) mx[k] = nm[k];
    i0 += 16;
  }
  const uint32_t fail = bias_logs(mx, lg);
  store(i0 - 16 - r0, fail);                     // the last batch may end in rows no one reads
  if (glane == 0) S.state[it] = make_float4(s0, s1, d0, d1);
}

// Groups of G lanes: the first cap_item of them a segment of a long sequence
// each, the others one listed sequence each.
template <int G, bool ONE>
__global__ void __launch_bounds__(128)
bias_kernel(BiasDev B, DbDev db, const int64_t *__restrict__ slots, const int64_t *__restrict__ order, int64_t nids,
            BiasSegs S, float *__restrict__ out, int32_t *__restrict__ out_len) {
  __shared__ BiasShared sh;
  const int lane = threadIdx.x & 31, glane = lane % G;
  const unsigned gmask = ((1u << G) - 1u) << (lane - glane);
  const int64_t g = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) / G;
  if ((int64_t) blockIdx.x * blockDim.x / G >= (int64_t) S.n[1] && ((int64_t) blockIdx.x + 1) * blockDim.x / G <= S.cap_item)
    return;                                      // a block past the last segment
  sh.load(B);
  if (g < S.cap_item) {
    if (g < S.n[1]) bias_segment<G, ONE>(B, sh, db, slots, S, (unsigned) g, glane);
    return;
  }
  const int64_t t = g - S.cap_item;
  if (t >= nids) return;
  const int64_t j = order[t];
  const int64_t s = slots[j];
  const int L = db.len[s];
  if (glane == 0) out_len[j] = L;
  if (L <= 0) { if (glane == 0) out[j] = 0.0f; return; }
  if (S.is_long[j]) return;
  const float sc = bias_score<G, ONE>(B, sh, reinterpret_cast<const uint4 *>(db.codes + db.start[s]), L, glane, gmask);
  if (glane == 0) out[j] = sc;
}

// One warp per long sequence: are its segments the sequence's own rows? Then
// the sum of the row logs in row order, by every lane alike; else its score
// from the start.
template <bool ONE>
__global__ void __launch_bounds__(128)
bias_join_kernel(BiasDev B, DbDev db, const int64_t *__restrict__ slots, BiasSegs S, float *__restrict__ out) {
  __shared__ BiasShared sh;
  const int lane = threadIdx.x & 31;
  if (blockIdx.x * (blockDim.x / 32) >= S.n[0]) return;
  sh.load(B);
  const unsigned e = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (e >= S.n[0]) return;
  const int j = S.seq[e];
  const int64_t s = slots[j];
  const int L = db.len[s], nseg = (L + kBiasSeg - 1) / kBiasSeg;
  const float4 *st = S.state + S.first[e];
  bool same = true;
  for (int k = lane + 1; k < nseg; k += 32)
    same = same && __float_as_uint(st[k].x) == __float_as_uint(st[k - 1].z) &&
           __float_as_uint(st[k].y) == __float_as_uint(st[k - 1].w);
  float sc;
  if (__all_sync(FULL, same)) {
    const float4 *lg = reinterpret_cast<const float4 *>(S.lg + (size_t) S.row[e] * kBiasSeg);
    float logsc = 0.0f;
    int r = 0;
    constexpr int U = 16;                        // 64 rows' loads ahead of their adds
    float4 v[U], nx[U];
#pragma unroll
    for (int u = 0; u < U; ++u) nx[u] = lg[u];   // a long sequence has more rows than these
    for (; r + 4 * U <= L; r += 4 * U) {
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = nx[u];
      if (r + 8 * U <= L) {
#pragma unroll
        for (int u = 0; u < U; ++u) nx[u] = lg[(r >> 2) + U + u];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        logsc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(logsc, v[u].x), v[u].y), v[u].z), v[u].w);
    }
    for (; r < L; ++r) logsc = __fadd_rn(logsc, reinterpret_cast<const float *>(lg)[r]);
    sc = __fadd_rn(logsc, log_rowf(__fadd_rn(st[nseg - 1].z, st[nseg - 1].w), sh.logtab));
  } else {
    sc = bias_score<16, ONE>(B, sh, reinterpret_cast<const uint4 *>(db.codes + db.start[s]), L, lane % 16,
                             lane < 16 ? 0xffffu : 0xffff0000u);
  }
  if (lane == 0) out[j] = sc;
}

// degenerate amino codes 21..26 (B J Z O U X) as sets of canonical codes
// (easel/esl_alphabet.c:282-292; X is every residue)
bool degen(int x, int y) {
  switch (x) {
    case 21: return y == 2 || y == 11;     // B: D N
    case 22: return y == 7 || y == 9;      // J: I L
    case 23: return y == 3 || y == 13;     // Z: E Q
    case 24: return y == 8;                // O: K
    case 25: return y == 1;                // U: C
    case 26: return true;                  // X
  }
  return false;
}

// esl_hmm_Configure (easel/esl_hmm.c:116-153) of the filter HMM with fq = bg->f
void filter_hmm(const float *compo, int M, BiasDev &B) {
  const float *bg = msvgb_detail::kAminoBg;
  const float *e[2] = {bg, compo};
  for (int x = 0; x < 20; ++x)
    for (int k = 0; k < 2; ++k) B.eo[x][k] = e[k][x] / bg[x];
  for (int k = 0; k < 2; ++k) B.eo[20][k] = B.eo[27][k] = B.eo[28][k] = 1.0f;
  for (int x = 21; x <= 26; ++x)
    for (int k = 0; k < 2; ++k) {
      float num = 0.0f, denom = 0.0f;
      for (int y = 0; y < 20; ++y)
        if (degen(x, y)) { num += e[k][y]; denom += bg[y]; }
      B.eo[x][k] = (denom > 0.0f) ? num / denom : 0.0f;
    }
  const float L1 = (float) ((double) M / 8.0);    // p7_bg_SetFilter: L1 = (float) M / 8.0
  B.t10 = 1.0f / (L1 + 1.0f);
  B.t11 = L1 / (L1 + 1.0f);
  B.pi0 = 0.999f;
  B.pi1 = 0.001f;
  for (int j = 0; j < kLogTab; ++j) {
    double c = 1.0 + (j + 0.5) / kLogTab;
    if (j >= 212) c *= 0.5;                         // f >= 1 + 212/512 is halved
    if (j == 0 || j == kLogTab - 1) c = 1.0;        // the intervals next to 1
    const double inv = 1.0 / c;
    B.logtab[j] = make_double2(inv, -std::log(inv));
  }
}

// Whether one division per row suffices (bias_kernel ONE): the background odds
// near 1 and the transitions out of either state positive, so that a row whose
// last maximum was either state's has a positive, finite maximum again.
bool one_division(const BiasDev &B) {
  for (int x = 0; x < NRES - 1; ++x)
    if (!(B.eo[x][0] >= 0.5f && B.eo[x][0] <= 2.0f && B.eo[x][1] >= 0.0f && B.eo[x][1] <= 1e30f)) return false;
  return B.t10 > 1e-30f && B.t10 <= 1.0f && B.t11 >= 0.0f && B.t11 <= 1.0f;
}

// Lanes per sequence: 4, 8 and 16 measured alike on 40,000 listed sequences
// (1.12, 1.08, 1.08 ms for the call): the longest sequence's chain decides.
constexpr int kBiasLanes = 8;

cudaError_t launch_bias(const BiasDev &B, const DbDev &db, const int64_t *ids, const int64_t *order, int64_t n,
                        const BiasSegs &S, float *out, int32_t *len, cudaStream_t stream) {
  constexpr int G = kBiasLanes;
  const unsigned grid = (unsigned) (((n + S.cap_item) * G + 127) / 128);
  const bool one = one_division(B);
  (void) cudaGetLastError();
  if (S.cap_row) bias_plan_kernel<<<(unsigned) ((n + 255) / 256), 256, 0, stream>>>(db, ids, n, S);
  if (one) bias_kernel<G, true><<<grid, 128, 0, stream>>>(B, db, ids, order, n, S, out, len);
  else bias_kernel<G, false><<<grid, 128, 0, stream>>>(B, db, ids, order, n, S, out, len);
  if (S.cap_row) {
    const unsigned joins = (S.cap_seq + 3) / 4;
    if (one) bias_join_kernel<true><<<joins, 128, 0, stream>>>(B, db, ids, S, out);
    else bias_join_kernel<false><<<joins, 128, 0, stream>>>(B, db, ids, S, out);
  }
  return cudaGetLastError();
}

}  // namespace

// The float-pair table of log_ff, uploaded once per device.
static cudaError_t ensure_logff(int device) {
  static std::mutex mu;
  static std::vector<int> done;
  std::lock_guard<std::mutex> lk(mu);
  for (int d : done) if (d == device) return cudaSuccess;
  std::vector<float4> t(2048);
  for (int j = 0; j < 2048; ++j) {
    double c = 1.0 + (j + 0.5) / 2048.0;
    if (j >= 849) c *= 0.5;
    if (j == 0 || j == 2047) c = 1.0;
    const double inv = 1.0 / c, lg = std::log(c);
    const float ih = (float) inv, th = (float) lg;
    t[j] = make_float4(ih, (float) (inv - (double) ih), th, (float) (lg - (double) th));
  }
  const cudaError_t e = cudaMemcpyToSymbol(g_logff, t.data(), sizeof(float4) * 2048);
  if (e == cudaSuccess) done.push_back(device);
  return e;
}

// p7_bg_FilterScore: nullsc + (float) L * logf(bg->p1) + logf(1. - bg->p1)
static float2 length_terms(int L) {
  const float p1 = (float) L / (float) (L + 1);
  return make_float2((float) L * logf(p1), logf((float) (1. - (double) p1)));
}

extern "C" float msvgb_bias_length_term(float fwd, int L) {
  const float2 t = length_terms(L);
  return fwd + t.x + t.y;
}

extern "C" int msvgb_stage_pass(float sc, float base, double mu, double lambda, double F, double *ret_P) {
  const float seq_score = (float) ((double) (sc - base) / 0.69314718055994529);
  const double y = lambda * ((double) seq_score - mu);
  const double ey = -exp(-y);
  const double P = (fabs(ey) < 5e-9) ? -ey : 1 - exp(ey);      // esl_gumbel_surv, easel/esl_gumbel.c:129-137
  if (ret_P) *ret_P = P;
  return (P > F) ? 0 : 1;
}

extern "C" float msvgb_null_score(int L) {
  const float p1 = (float) L / (float) (L + 1);                  // p7_bg_NullOne, src/p7_bg.c:359-363
  return (float) ((double) (float) L * ::log((double) p1) + ::log(1. - (double) p1));
}

extern "C" int msvgb_biasfilter(msvgb_ctx *c, const float *compo, int M, const msvgb_db *db, const int64_t *ids,
                                int64_t nids, float *out_sc) {
  if (!c || !compo || !db || M < 1 || nids < 0 || (nids && (!ids || !out_sc)))
    return fail(MSVGB_eslEINVAL, "msvgb_biasfilter: bad arguments");
  if (nids == 0) return MSVGB_eslOK;
  for (int64_t j = 0; j < nids; ++j)
    if (ids[j] < 0 || ids[j] >= db->n) return fail(MSVGB_eslEINVAL, "sequence index out of range");
  CUDA_TRY(cudaSetDevice(c->device));
  BiasDev B;
  filter_hmm(compo, M, B);
  CUDA_TRY(ensure_logff(c->device));
  CUDA_TRY(msvgb_detail::ensure_inverse(c, db));
  // one scratch block: list slots and order (int64), bucket counts, scores and lengths
  const size_t a8 = ((size_t) nids * 8 + 255) & ~(size_t) 255, a4 = ((size_t) nids * 4 + 255) & ~(size_t) 255;
  char *d_scr = nullptr;
  cudaMemPool_t pool = msvgb_detail::scratch_pool(c->device);   // stays mapped between calls
  if (!pool) return fail(MSVGB_eslESYS, "biasfilter: no memory pool");
  // room for the long sequences: at most 4M rows of them at a time, and no more than the list can hold
  BiasSegs S{};
  const int64_t most = db->Lmax > kBiasLong ? nids * ((db->Lmax + kBiasSeg - 1) / kBiasSeg) : 0;
  S.cap_row = (unsigned) std::min<int64_t>(most, (4 << 20) / kBiasSeg);
  S.cap_item = S.cap_row;
  S.cap_seq = (unsigned) std::min<int64_t>(nids, S.cap_row / 3);   // a long one has four segments or more
  size_t end = 2 * a8 + 4096 + 2 * a4;
  auto take = [&](size_t bytes) { const size_t at = end; end += (bytes + 255) & ~(size_t) 255; return at; };
  const size_t o_long = take((size_t) nids), o_n = take(12), o_item = take((size_t) S.cap_item * 8),
               o_state = take((size_t) S.cap_item * 16), o_lg = take((size_t) S.cap_row * kBiasSeg * 4),
               o_seq = take((size_t) S.cap_seq * 12);
  CUDA_TRY(cudaMallocFromPoolAsync((void **) &d_scr, end, pool, c->stream));
  S.is_long = (uint8_t *) d_scr + o_long;
  S.n = (unsigned *) (d_scr + o_n);
  S.item = (uint2 *) (d_scr + o_item);
  S.state = (float4 *) (d_scr + o_state);
  S.lg = (float *) (d_scr + o_lg);
  S.seq = (int32_t *) (d_scr + o_seq);
  S.first = (unsigned *) S.seq + S.cap_seq;
  S.row = S.first + S.cap_seq;
  int64_t *d_ids = (int64_t *) d_scr, *d_order = (int64_t *) (d_scr + a8);
  int32_t *d_cnt = (int32_t *) (d_scr + 2 * a8);
  float *d_out = (float *) (d_scr + 2 * a8 + 4096);
  int32_t *d_len = (int32_t *) (d_scr + 2 * a8 + 4096 + a4);
  // ids up and results back through pinned scratch (pageable copies may run as kernels)
  uint8_t *pin = msvgb_detail::pinned_scratch(c, a8 + 2 * a4);
  if (!pin) { cudaFreeAsync(d_scr, c->stream); return fail(MSVGB_eslEMEM, "biasfilter: pinned scratch"); }
  memcpy(pin, ids, (size_t) nids * 8);
  cudaError_t e = cudaMemcpyAsync(d_ids, pin, nids * 8, cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = msvgb_detail::launch_gather_ids(d_ids, nids, db->d_inv, c->num_sms, c->stream);
  if (e == cudaSuccess)
    e = msvgb_detail::launch_order_by_length(d_ids, nids, db->d_len, db->Lmax, d_cnt, d_order, c->num_sms, c->stream);
  DbDev dbv{db->d_codes, db->d_start, db->d_len, db->d_orig, db->n};
  if (e == cudaSuccess) e = cudaMemsetAsync(d_scr + o_long, 0, o_n + 12 - o_long, c->stream);   // is_long, n
  if (e == cudaSuccess) e = launch_bias(B, dbv, d_ids, d_order, nids, S, d_out, d_len, c->stream);
  if (e == cudaSuccess) msvgb_detail::count_launch();
  const float *sc = (const float *) (pin + a8);                  // scores, then lengths, in one copy
  const int32_t *lens = (const int32_t *) (pin + a8 + a4);
  if (e == cudaSuccess) e = cudaMemcpyAsync(pin + a8, d_out, a4 + (size_t) nids * 4, cudaMemcpyDeviceToHost, c->stream);
  cudaFreeAsync(d_scr, c->stream);
  const cudaError_t e2 = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) return fail(MSVGB_eslESYS, std::string("biasfilter: ") + cudaGetErrorString(e));
  // the length terms, one pair of logarithms per length (L logf(p1), then logf(1 - p1), as
  // msvgb_bias_length_term adds them); the few lengths past kTerms each time
  constexpr int kTerms = 1 << 16;
  std::vector<float2> term((size_t) std::min(db->Lmax, kTerms) + 1, make_float2(NAN, 0.0f));
  for (int64_t j = 0; j < nids; ++j) {
    const int L = lens[j];
    if (L <= 0) { out_sc[j] = 0.0f; continue; }
    float2 past = make_float2(NAN, 0.0f);
    float2 &t = L <= kTerms ? term[L] : past;
    if (std::isnan(t.x)) t = length_terms(L);
    out_sc[j] = sc[j] + t.x + t.y;
  }
  return MSVGB_eslOK;
}
