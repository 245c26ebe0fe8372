// resident.cuh -- the block-resident decoder: one launch for all iterations, a CTA per task.
//
// A task is one or more whole code blocks, one thread per window, and a CTA keeps it from the
// first half-iteration to the last: the LLR that every half-iteration reads (Ls + the other SISO's
// extrinsic) stays in shared memory for the whole decode, in natural order, so neither SISO needs
// an interleaved copy and no half-iteration waits for another CTA.  The streams that are only read
// (parities, systematic) and the alpha checkpoints sit in a scratch slot per resident CTA, laid
// out so that the lanes of a warp access consecutive words; the slots are reused from task to task.
// With all SMs full they are larger than L2 (246 MB at windows of 192) and are partly read from DRAM again.
//
// Arithmetic: the state metrics are kept as probabilities (float32, scaled by powers of two), not
// as logarithms.  A trellis step of the 8 states is 16 multiply-adds and two ex2 for the branch
// weights, where the (m, s) form of trellis.cuh needs 8 ex2 and about 85 instructions; the
// extrinsic is one lg2 of each of two 4-term sums.  What limits it is float's exponent range: a
// probability below 2^-149 becomes 0.  Each half-iteration checks, per block, that what was lost cannot
// matter (kLost below).  A block whose LLRs leave the range of one weight per input (126 bits) or whose
// checks come close goes on in a two-factor form of the same arithmetic, and from there, if it has to, in
// the (m, s) form (siso.cuh), in passes of their own.  LLRs of ordinary channels stay
// inside the linear range (extrinsics of about 120 to 170 bits, depending on the parities; eight
// iterations at 1/3 reach 90 bits at 1 dB, 143 at 2.5 dB); blocks of rate 4/5 that fail their CRC may
// leave it, scaled-up LLRs do.
//
// The linear passes keep all LLRs in base-2 units (natural LLR * log2(e)).
//
// What bounds it: the issue slots of the SMs, at 2 warps per scheduler (about 131 instructions per step of a
// half-iteration, warm-ups included, 161 before most multiplications and multiply-adds went in pairs; the
// (m, s) form has about 450).  One warp of 32 windows of 192 steps per CTA, because the shared memory of an
// SM holds X of 8 of them (7 CTAs with rows of 33 words and a ring of 4 stages were 4 % slower).  4096
// blocks of K = 6144, 8 iterations: 2.69 ms, 8.0 ms with the (m, s) kernel that this one replaced.  One block
// of K = 6144 from host memory: 0.42 ms (1.08 ms); 20000 mixed blocks with early stop: 5.9 ms (14.3 ms).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "decoder.hpp"
#include "siso.cuh"

namespace tcb {
namespace {

constexpr int kResMaxX = 65536 - 256;             // bytes of X: its offsets are 16 bits
constexpr int kResMaxSmem = 227 * 1024;
constexpr uint64_t kWaitLimitNs = 1000000000ull;  // of a device-side wait: one second

// One code block as the kernel sees it; the blocks of a task are consecutive in the list.
struct ResCb {
  int32_t k, filler;
  int32_t tab;     // offset of this K's permutation table
  int32_t lane0;   // thread of the block's first window within its task
  int32_t nwin, window;
  int32_t idx;     // the caller's index of the block (flags, iteration counts)
  int32_t pad;
  int64_t llr;     // float offset of [d0|d1|d2]
  int64_t out;     // float offset of the posterior
};

struct ResArgs {
  const ResCb* cbs;
  const int32_t* task_first;  // [n_tasks + 1]: first block of each task
  int n_tasks;
  int* queue;                 // next task beyond the grid (zero before the launch)
  const int* never;           // testing hook: a word that stays 0
  int* error;
  int stall_task;             // testing hook (-1: off)
  const float* llr;
  float* post;
  const uint16_t* perm;
  const uint32_t* xpow;       // x^j mod g_CRC24B, kXpowSize entries, then b(x) x^24 mod g per byte b
  float4* scratch;
  int64_t slot;               // float4 per scratch slot (one slot per CTA of the grid)
  int guard;
  int max_iterations;
  int early_stop;
  uint8_t* crc_ok;
  uint32_t* iters;
  const float* scale;         // [2 * max_iterations]
};

__device__ __forceinline__ int load_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Scratch slot of a CTA, in planes of a float4 per thread or, in the compact layout, per window of the
// task (rows8 = longest window / 8, one record per 8 steps):
//   upper SISO: rows8 records of parity 1 (2 planes), the shared-memory byte offsets of the 8
//     positions (8 x uint16: 1), systematic (2)
//   lower SISO: the same of parity 2 and the interleaved positions
//   alpha checkpoints, one per 8 steps (the extrinsics of the 8 steps replace it): 2 rows8
//   what the half-iteration read, for an (m, s) pass that takes over from there: 2 rows8
//   ((m, s) pass: behind the extrinsics, checkpoints of the (m, s) form, one per 4 steps, and one
//   more): 4 rows8 + 2
//   seeds: 2 SISOs x 2 iteration parities x (alpha, beta) x 2 planes: 16
//   beta at the block end (log values) of the upper and the lower SISO: 4
// and the windows behind them (k, window, nwin, lane0: 4 x uint16, in one float4 per thread).
// Both SISOs take their places in X from the record, so that they share one copy of the code (with a
// copy each, the phases that the warps of an SM are in at a time overflow the instruction cache).
__host__ __device__ inline int64_t res_slot(int threads, int rows8, int pitch) {  // in float4
  return (16 * static_cast<int64_t>(rows8) + 22) * pitch + threads;
}
// An instance of the kernel.  The compact layout is for one warp with few long windows: X leaves room for
// 6144 steps of a warp, so a block of full-length windows has one lane of 32 in use, and planes of 32 would
// take 6.3 MB a CTA, 7.5 GB in all (0.2 MB and 0.23 GB compact).  Its pitch is a run-time value, which the
// short windows do without: their loops take the planes' offsets as constants.
template <int THREADS, bool COMPACT>
struct Shape {
  static constexpr int kThreads = THREADS;
  static constexpr bool kCompact = COMPACT;
};

// Scaling and checks.  The branch weights of a step are below 2, so that the largest metric grows by at
// most 3 per step; every 8 steps it is set to 2^top, as high as the block's largest parity weight
// leaves room for in the products (res_top).  What falls below float's range is an absolute error of
// 2^-150 in a metric: a path cut off there weighs at most 2^-150 2^(top + 13) of a mass of all paths (the
// sum of alpha beta, the same throughout a group of 8 steps).  The smaller side of an extrinsic x has
// 2^-|x| of the mass and must be 2^kKept times what was lost anywhere in the block (half an ulp of
// an x of 64 or more), so that a block passes if
//   log2(smallest mass) - max |x| >= top + 13 - 150 + kKept.
// That holds as long as it is metrics that lose, never weights (a lost weight counts relative to metrics
// of up to 2^top), and as long as nothing grows again that was lost.  So, with q = log2 of the largest parity
// weight or of its inverse (weights below 2^-kVoid left out, see the first point):
// - While every weight is above 2^-126 the unlikely input's weight is one factor (the plain form).  A block
//   in which one is not, which alpha finds out before X changes, or that is within kNearPlain of the limit
//   changes to two factors of 2^(-|s| / 2) applied to the metrics one after the other (WideWeights).  They are
//   0 from 252 bits on, where the product with a metric, below 2^(top + 15), is far below 2^-150 in any case;
//   so is a parity weight below 2^-kVoid.  (Infinite LLRs of known bits are exact: weights of 0 that lose
//   nothing.)  The two-factor form takes half as long again: the change comes as late as is safe (a bound of |s|
//   from the systematic LLR's and the extrinsics' maxima instead of the weights themselves: 4096 blocks of K =
//   6144 at 2 dB 3.5 ms instead of 3.0, 20000 of K = 512 at 3 dB 3.4 instead of 2.7).
// - beta multiplies by the input weights first, the power of two of `weights` among them, and by the
//   parity weight then, up to 2^q: the plain form leaves q bits less.  (The two-factor form applies the power
//   of two behind the parity; the TS 36.212 code has one product per branch.)
// - The x of a step leaves out that step's own input weight, and paths that only this weight made
//   negligible can be all of one side of x.  That takes evidence on the neighbouring steps against this
//   weight, which shows as a fall of the largest metric: what it falls by within a group beyond kKept bits is
//   taken off too (falls stay below 20 bits on codewords; blocks that this had to catch had 60 and more).
// Shown by a restatement on the CPU, 3.2 million blocks of codewords and of noise (AWGN, fading, punctured,
// saturated and independent LLRs of up to 200 bits, both codes), every half-iteration against 64 bits: those
// that passed were within 1.1e-5 max(|x + s|, 1 nat).  One factor throughout and neither deduction: off by up
// to 18 bits.
constexpr int kKept = 18;
// A block of the two-factor form that is within kNear of failing keeps what its half-iterations read, so that
// the (m, s) pass can go on there (a store more per step); one that fails from further off starts again.
constexpr float kNear = 40.0f;
constexpr float kNearPlain = 30.0f;  // (24: some blocks fail all at once and start again, 512 transport blocks 7 % slower)
constexpr float kLost = 150.0f - 13.0f - kKept;
constexpr float kMaxParity = 76.0f;  // larger ones (of either sign, but for the void) go to the (m, s) pass at once
constexpr float kVoid = 230.0f;      // 150 bits and those of the largest product of a metric and a weight
constexpr int kTopMax = 60;
// top of a block whose largest parity weight is 2^q: leaves the products of a step 18 bits of growth
// below 2^126 (on ordinary channels alpha and beta grow by 4 or 5 each)
__device__ __forceinline__ int res_top(float q) {
  return min(kTopMax, static_cast<int>(0.5f * (108.0f - fminf(q, kMaxParity))));
}

// min(x, y, z) of what is not NaN; min(x, y), max(x, y, z), NaN if any is
__device__ __forceinline__ float min3(float x, float y, float z) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
  return r;
}
__device__ __forceinline__ float min_nan(float x, float y) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float max3_nan(float x, float y, float z) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
  return r;
}

// Branch weights of one step from s = log2(e) (Ls + La) and b = 2^(log2(e) Lp): input 1 / input 0 and
// parity 1 (parity 0: 1).  The input weights carry the power of two that keeps the likeliest branch
// below 2.  (2^(log2(e) Lp) is in the record: a step needs one ex2 here, not two or three, and the
// unit that computes it was busy for half of the time.)
struct Weights {
  static constexpr bool kWide = false;
  float a1, a0, b;
  float x;  // the smaller of a1, a0
};
__device__ __forceinline__ float weight_scale(float b) {
  return __int_as_float(0x7f000000 - (__float_as_int(fmaxf(b, 1.0f)) & 0x7f800000));
}
__device__ __forceinline__ void weights(float s, float b, Weights& w) {
  const float y = weight_scale(b);
  const float x = ex2(-fabsf(s)) * y;
  w = Weights{s < 0.0f ? x : y, s < 0.0f ? y : x, b, x};
}
// The same in the two-factor form: input 1 / input 0 are c1^2 y / c0^2 y, y the power of two and c of the
// unlikely input 2^(-|s| / 2).
struct WideWeights {
  static constexpr bool kWide = true;
  float c1, c0, y, b;
};
__device__ __forceinline__ void weights(float s, float b, WideWeights& w) {
  const float h = ex2(-0.5f * fabsf(s));
  w = WideWeights{s < 0.0f ? h : 1.0f, s < 0.0f ? 1.0f : h, weight_scale(b), b};
}

// log2(x / y) of positive normal x, y (y < 2^126): the exponents' difference is exact and what is left
// of the ratio is in [1, 2), so that the result is rounded once at its own size.  (lg2 of each side,
// of the size of the scaled metrics, is 6 instructions shorter and 3 times further off.)
__device__ __forceinline__ float log_ratio(float x, float y) {
  const int d = (__float_as_int(x) - __float_as_int(y)) & 0xff800000;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  const float e = __int_as_float((d >> 23) + 0x4b400000) - 12582912.0f;  // d 2^-23
  return e + lg2(__int_as_float(__float_as_int(x) - d) * r);
}

// The scale 2^(top - exponent of the largest of m).
__device__ __forceinline__ float rescale(const float (&m)[8], int top) {
  const float x = max3(max3(m[0], m[1], m[2]), max3(m[3], m[4], m[5]), max3(m[6], m[7], 0x1p-60f));
  return __int_as_float(((top + 254) << 23) - (__float_as_int(x) & 0x7f800000));
}

// Reference code: at[n] = sum over the two branches into n of alpha * parity weight; the input
// weight is common to both (pred_input depends on n only) and is applied by alpha_scale.
__device__ __forceinline__ void alpha_lin(const float (&al)[8], float b, float (&at)[8]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x = al[2 * j], y = al[2 * j + 1];
    const float u = fmaf(b, y, x), v = fmaf(b, x, y);
    at[j] = j < 2 ? u : v;
    at[j + 4] = j < 2 ? v : u;
  }
}
__device__ __forceinline__ void input_scale(const float (&at)[8], float a1, float a0, float (&al)[8]) {
#pragma unroll
  for (int n = 0; n < 8; ++n) al[n] = at[n] * (pred_input<false>(n, 0) ? a1 : a0);
}
// beta_t from beta_{t+1} times the input weights
__device__ __forceinline__ void beta_lin(const float (&bh)[8], float b, float (&be)[8]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x = bh[j], y = bh[j + 4];
    const float u = fmaf(b, y, x), v = fmaf(b, x, y);
    be[2 * j] = j < 2 ? u : v;
    be[2 * j + 1] = j < 2 ? v : u;
  }
}
// The TS 36.212 code: both input and parity weights differ between the branches into a state.
__device__ __forceinline__ void std_weights(const Weights& w, float (&g)[2][2]) {
  g[0][0] = w.a0;
  g[0][1] = w.a0 * w.b;
  g[1][0] = w.a1;
  g[1][1] = w.a1 * w.b;
}
__device__ __forceinline__ void alpha_std(const float (&al)[8], const float (&g)[2][2], float (&out)[8]) {
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const int p0 = 2 * (n & 3);
    out[n] = fmaf(al[p0], g[pred_input<true>(n, 0)][pred_parity(n, 0)],
                  al[p0 + 1] * g[pred_input<true>(n, 1)][pred_parity(n, 1)]);
  }
}
__device__ __forceinline__ void beta_std(const float (&be)[8], const float (&g)[2][2], float (&out)[8]) {
#pragma unroll
  for (int s = 0; s < 8; ++s)
    out[s] = fmaf(be[next_state<true>(s, 0)], g[0][parity<true>(s, 0)],
                  be[next_state<true>(s, 1)] * g[1][parity<true>(s, 1)]);
}

// Packed pairs (fma.rn.f32x2 and mul.rn.f32x2: one issue slot for two operations, each rounded as the
// scalar one, so that the results are bit for bit the same).  The reference code's recursions use them,
// because issue slots are what the kernel runs out of: 4096 blocks of K = 6144 2892 -> 2800 us, 512 of them
// with early stop 511 -> 488 us, 20000 mixed blocks 6797 -> 6167 us, 1000 of K = 1024 383 -> 355 us.  (In
// lin_read alone: 2923 us where the whole takes 2728.)  The TS 36.212 code has 4 products of weights per
// step that differ between the branches into a state, and stays scalar.
__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t p, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(p));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// The branches of the reference code with parity 0: the predecessor of state n, and its inverse.  The
// branches with parity 1 come from unit_pred(n) ^ 1 and go to unit_succ(p) ^ 4.
__host__ __device__ constexpr int unit_pred(int n) {
  return (n >> 1 & 1) << 2 | (n & 1) << 1 | ((n >> 2 ^ n >> 1) & 1);
}
__host__ __device__ constexpr int unit_succ(int p) {
  return ((p >> 2 ^ p) & 1) << 2 | (p >> 2 & 1) << 1 | (p >> 1 & 1);
}
// alpha_lin, beta_lin and input_scale on the pairs (s, s ^ M) of the states s without bit F; the results
// are the pairs of unit_succ (alpha) or unit_pred (beta) of these.
template <int M, int F>
__device__ __forceinline__ void alpha_lin2(const float (&al)[8], float b, float (&at)[8]) {
  const uint64_t bb = pack2(b, b);
#pragma unroll
  for (int s = 0; s < 8; ++s)
    if ((s & F) == 0)
      unpack2(fma2(bb, pack2(al[s ^ 1], al[s ^ 1 ^ M]), pack2(al[s], al[s ^ M])), at[unit_succ(s)],
              at[unit_succ(s ^ M)]);
}
template <int M, int F>
__device__ __forceinline__ void beta_lin2(const float (&bh)[8], float b, float (&be)[8]) {
  const uint64_t bb = pack2(b, b);
#pragma unroll
  for (int s = 0; s < 8; ++s)
    if ((s & F) == 0)
      unpack2(fma2(bb, pack2(bh[s ^ 4], bh[s ^ 4 ^ M]), pack2(bh[s], bh[s ^ M])), be[unit_pred(s)],
              be[unit_pred(s ^ M)]);
}
template <int M, int F>
__device__ __forceinline__ void input_scale2(const float (&at)[8], float a1, float a0, float (&al)[8]) {
#pragma unroll
  for (int s = 0; s < 8; ++s)
    if ((s & F) == 0)
      unpack2(mul2(pack2(at[s], at[s ^ M]), pack2(pred_input<false>(s, 0) ? a1 : a0, pred_input<false>(s ^ M, 0) ? a1 : a0)),
              al[s], al[s ^ M]);
}

// Step t of a group of 8.  The pairs of one step are the operands of the next one, in the same order of
// their two states, for two steps; in the third the orders of the two operands differ (the map has no
// functional that stays 0 on three parity branches), and the scalar step, which reads and leaves its
// values in any register, brings back the first pairs.
__device__ __forceinline__ void alpha_lin_at(int t, const float (&al)[8], float b, float (&at)[8]) {
  if (t % 3 == 0) alpha_lin2<4, 4>(al, b, at);
  else if (t % 3 == 1) alpha_lin2<6, 2>(al, b, at);
  else alpha_lin(al, b, at);
}
__device__ __forceinline__ void alpha_scale_at(int t, const float (&at)[8], float a1, float a0, float (&al)[8]) {
  if (t % 3 == 0) input_scale2<6, 2>(at, a1, a0, al);
  else if (t % 3 == 1) input_scale2<7, 1>(at, a1, a0, al);
  else input_scale2<4, 4>(at, a1, a0, al);
}
__device__ __forceinline__ void beta_scale_at(int t, const float (&be)[8], float a1, float a0, float (&x)[8]) {
  const int phase = (7 - t) % 3;
  if (t == 7) input_scale(be, a1, a0, x);  // the group before left other pairs
  else if (phase == 0) input_scale2<1, 1>(be, a1, a0, x);
  else if (phase == 1) input_scale2<2, 2>(be, a1, a0, x);
  else input_scale2<5, 4>(be, a1, a0, x);
}
__device__ __forceinline__ void beta_lin_at(int t, const float (&x)[8], float b, float (&out)[8]) {
  const int phase = (7 - t) % 3;
  if (phase == 0) beta_lin2<1, 1>(x, b, out);
  else if (phase == 1) beta_lin2<2, 2>(x, b, out);
  else beta_lin(x, b, out);
}

__device__ __forceinline__ void scale_all(float (&m)[8], float r) {
  const uint64_t rr = pack2(r, r);
#pragma unroll
  for (int s = 0; s < 8; s += 2) unpack2(mul2(pack2(m[s], m[s + 1]), rr), m[s], m[s + 1]);
}
// alpha's input weights; one alpha step with weights w, one beta step with weights w of metrics to be scaled
// by r before the group's first: step t of a group.
__device__ __forceinline__ void alpha_input(int step, const float (&at)[8], const Weights& w, float (&al)[8]) {
  alpha_scale_at(step, at, w.a1, w.a0, al);
}
template <bool STD>
__device__ __forceinline__ void alpha_next(int step, float (&al)[8], const Weights& w) {
  float t[8];
  if constexpr (STD) {
    float g[2][2];
    std_weights(w, g);
    alpha_std(al, g, t);
#pragma unroll
    for (int n = 0; n < 8; ++n) al[n] = t[n];
  } else {
    alpha_lin_at(step, al, w.b, t);
    alpha_scale_at(step, t, w.a1, w.a0, al);
  }
}
template <bool STD>
__device__ __forceinline__ void beta_next(int step, float (&be)[8], const Weights& w, float r) {
  float t[8];
  if (step == 7) scale_all(be, r);
  if constexpr (STD) {
    float g[2][2];
    std_weights(w, g);
    beta_std(be, g, t);
#pragma unroll
    for (int n = 0; n < 8; ++n) be[n] = t[n];
  } else {
    float x[8];
    beta_scale_at(step, be, w.a1, w.a0, x);
    beta_lin_at(step, x, w.b, t);
#pragma unroll
    for (int n = 0; n < 8; ++n) be[n] = t[n];
  }
}
// The smallest weight of two steps (the TS 36.212 code: or product of weights) and `least`.
template <bool STD>
__device__ __forceinline__ float least_of(float least, const Weights& v, const Weights& w) {
  least = min3(least, v.x, w.x);
  return STD ? min3(least, v.x * v.b, w.x * w.b) : least;
}
template <bool STD>
__device__ __forceinline__ float least_of(float least, const WideWeights&, const WideWeights&) {
  return least;
}
// The mass of all paths from the sums of alpha beta over the branches with input 1 and 0.
__device__ __forceinline__ float mass_of(const Weights& w, float s1, float s0) { return fmaf(w.a1, s1, w.a0 * s0); }

// The two-factor form, factor by factor on the metrics, so that no product of weights is formed; the
// power of two comes behind the parity.  (In pairs like the plain form; without them 512 transport blocks took
// 60 us longer, mean of 8 batches.)
__device__ __forceinline__ void alpha_input(int step, const float (&at)[8], const WideWeights& w, float (&al)[8]) {
  alpha_scale_at(step, at, w.y, w.y, al);
  alpha_scale_at(step, al, w.c1, w.c0, al);
  alpha_scale_at(step, al, w.c1, w.c0, al);
}
__device__ __forceinline__ float wide_branch(float m, int input, int par, const WideWeights& w) {
  if (par) m *= w.b;
  const float c = input ? w.c1 : w.c0;
  return m * w.y * c * c;
}
template <bool STD>
__device__ __forceinline__ void alpha_next(int step, float (&al)[8], const WideWeights& w) {
  float t[8];
  if constexpr (STD) {
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int p0 = 2 * (n & 3);
      t[n] = wide_branch(al[p0], pred_input<true>(n, 0), pred_parity(n, 0), w) +
             wide_branch(al[p0 + 1], pred_input<true>(n, 1), pred_parity(n, 1), w);
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) al[n] = t[n];
  } else {
    alpha_lin_at(step, al, w.b, t);
    alpha_input(step, t, w, al);
  }
}
template <bool STD>
__device__ __forceinline__ void beta_next(int step, float (&be)[8], const WideWeights& w, float r) {
  float t[8];
  if (step == 7) scale_all(be, r);
  if constexpr (STD) {
#pragma unroll
    for (int s = 0; s < 8; ++s)
      t[s] = wide_branch(be[next_state<true>(s, 0)], 0, parity<true>(s, 0), w) +
             wide_branch(be[next_state<true>(s, 1)], 1, parity<true>(s, 1), w);
  } else {
    float x[8];
    beta_scale_at(step, be, w.c1, w.c0, x);
    beta_scale_at(step, x, w.c1, w.c0, x);
    beta_lin_at(step, x, w.b, t);
    scale_all(t, w.y);
  }
#pragma unroll
  for (int n = 0; n < 8; ++n) be[n] = t[n];
}
__device__ __forceinline__ float mass_of(const WideWeights& w, float s1, float s0) {
  return fmaf(w.y * s1 * w.c1, w.c1, w.y * s0 * w.c0 * w.c0);
}

// log2 metrics (largest 0) <-> scaled probabilities, down to float's smallest (ex2 and lg2 flush
// what is below 2^-126)
__device__ __forceinline__ void lin_from_log(const float (&v)[8], float (&m)[8], int top) {
  const float x = static_cast<float>(top + 24) - max8(v);
#pragma unroll
  for (int k = 0; k < 8; ++k) m[k] = 0x1p-24f * ex2(v[k] + x);
}
__device__ __forceinline__ void log_from_lin(const float (&m)[8], float (&v)[8]) {
  float r[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) r[k] = fmaxf(lg2(0x1p24f * m[k]), kNegBig);
  const float x = max8(r);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = fmaxf(r[k] - x, kNegBig);
}

// The phases of a decode are functions of their own (not inlined: in one function their address
// arithmetic is hoisted out of the iteration loops and spilled), so what they need is kept in shared
// memory: the CTA's constants and, per thread, its window.
// Words between the rows of X: the warp's windows in consecutive banks.  An odd number keeps the columns
// (inputs and outputs) free of bank conflicts too; full warps do without, because 8 CTAs of 32
// windows of 192 steps then fit in an SM.
__host__ __device__ inline int res_pitch(int lanes) { return lanes % 32 == 0 ? lanes : lanes | 1; }
struct ResCta {
  char* slot;          // the CTA's scratch slot
  int guard;
  int rows8;           // longest window of the task / 8
  uint32_t plane;      // (compact) bytes of a plane of the slot
  uint32_t xs4;        // bytes between the rows of X
  int max_window;      // of the task
  int next_task;
  uint32_t crc_tab[16];  // b(x) x^24 mod g of the 4-bit b
};
// Dynamic shared memory of a CTA: ResCta; a word per thread, used at the first thread of a
// block (kWordPar); the ring; X.  Between two passes over the streams the ring is idle, and four words per
// thread in it (kWordExt ..) pass a half-iteration's checks and the CRC between the block's threads.
extern __shared__ __align__(16) char res_smem[];
constexpr int kResHead = (sizeof(ResCta) + 15) / 16 * 16;
// Streams of the slot come through a ring in shared memory (cp.async, each thread its own
// entries), because the slots of all resident CTAs together are larger than L2: a group of 8 steps is
// requested two groups before its use, which covers most of a DRAM access without holding registers.  Stage: entries of 16 bytes per thread, [entry][thread].
constexpr int kStages = 2;
constexpr int kEntries = 3;  // of a stage: 2 of parity, 1 of positions
__host__ __device__ constexpr int res_ring_at(int nt) { return kResHead + 4 * nt; }
__host__ __device__ constexpr int res_x_at(int nt) { return res_ring_at(nt) + 16 * kStages * kEntries * nt; }

// What one thread knows of its window.
struct ResWin {
  int k, w, nwin, lo, len;   // block size, window, windows, first step, steps
  int window, guard;
  int tid, lane0;
  int prev, next;            // columns of the neighbouring windows (own column at the block ends)
  uint32_t xs4;
  int top;                   // of the block
};
__device__ __forceinline__ ResCta& res_cta() { return *reinterpret_cast<ResCta*>(res_smem); }
template <class S>
__device__ __forceinline__ ushort4* res_window() {
  const ResCta& c = *reinterpret_cast<const ResCta*>(res_smem);
  return reinterpret_cast<ushort4*>(c.slot + (16 * c.rows8 + 22) * (S::kCompact ? c.plane : 16u * S::kThreads));
}
// word `i` of the per-thread words
template <class S>
__device__ __forceinline__ int* res_word(int i) {
  return reinterpret_cast<int*>(res_smem + kResHead + 4 * S::kThreads * i);
}
constexpr int kWordPar = 0;   // largest |log2 parity weight|
// largest extrinsic, smallest mass, CRC, largest fall of alpha
constexpr int kWordExt = 1, kWordMass = 2, kWordSyn = 3, kWordFall = 4;
// the passes over a task
constexpr int kPlain = 0, kWide = 1, kLog = 2;
template <class S>
__device__ __forceinline__ char* res_x() {
  return res_smem + res_x_at(S::kThreads);
}
template <class S>
__device__ __forceinline__ ResWin res_win() {
  const ResCta& c = res_cta();
  const ushort4 t = res_window<S>()[threadIdx.x];
  ResWin v;
  v.tid = threadIdx.x;
  v.k = t.x;
  v.window = t.y;
  v.nwin = t.z;
  v.lane0 = t.w;
  v.w = v.tid - v.lane0;
  v.lo = v.w * v.window;
  v.len = min(v.window, v.k - v.lo);
  v.guard = c.guard;
  v.prev = v.w > 0 ? v.tid - 1 : v.tid;
  v.next = v.w + 1 < v.nwin ? v.tid + 1 : v.tid;
  v.xs4 = c.xs4;
  v.top = res_top(__int_as_float(res_word<S>(kWordPar)[v.lane0]));
  return v;
}

__device__ __forceinline__ float lds(const char* x, uint32_t off) {
  return *reinterpret_cast<const float*>(x + off);
}

// The scratch slot of the CTA, addressed by 32-bit byte offsets.  Plain loads and stores: what other
// lanes wrote is read after a barrier, never through the read-only path.
template <class S, bool = S::kCompact>
struct PlanePitch {
  static constexpr uint32_t plane = 16u * S::kThreads;
};
template <class S>
struct PlanePitch<S, true> {
  uint32_t plane;
  __device__ __forceinline__ PlanePitch() : plane(res_cta().plane) {}
};
template <class S>
struct Slot : PlanePitch<S> {
  using PlanePitch<S>::plane;
  char* base;
  uint32_t rows8;
  __device__ __forceinline__ Slot() : base(res_cta().slot), rows8(res_cta().rows8) {}
  // byte offset of an 8-step record of the upper / lower SISO, of the checkpoint of such a group, of
  // the seeds of a SISO written in iterations of a parity, of a SISO's tail
  __device__ __forceinline__ uint32_t record(bool lower, int g) const {
    return (lower ? rows8 : 0) * (5 * plane) + g * (5 * plane);
  }
  __device__ __forceinline__ uint32_t ckpt(int g) const { return (10 * rows8 + 2 * g) * plane; }
  // (two-factor form) what the last half-iteration read, 8 steps
  __device__ __forceinline__ uint32_t kept(int g) const { return (12 * rows8 + 2 * g) * plane; }
  __device__ __forceinline__ uint32_t seeds(bool lower, int it) const {
    return (16 * rows8 + 2 + (lower ? 8 : 0) + (it & 1 ? 4 : 0)) * plane;
  }
  __device__ __forceinline__ uint32_t tail(bool lower) const {
    return (16 * rows8 + 18 + (lower ? 2 : 0)) * plane;
  }
  // planes of a record
  __device__ __forceinline__ uint32_t index() const { return 2 * plane; }
  __device__ __forceinline__ uint32_t sys() const { return 3 * plane; }
  __device__ __forceinline__ float4 ld(uint32_t o) const { return *reinterpret_cast<const float4*>(base + o); }
  __device__ __forceinline__ uint2 ld2(uint32_t o) const { return *reinterpret_cast<const uint2*>(base + o); }
  __device__ __forceinline__ void st(uint32_t o, float4 v) const { *reinterpret_cast<float4*>(base + o) = v; }
  __device__ __forceinline__ void st2(uint32_t o, uint2 v) const { *reinterpret_cast<uint2*>(base + o) = v; }
  __device__ __forceinline__ void ld8(uint32_t o, float (&v)[8]) const {
    const float4 x = ld(o), y = ld(o + plane);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
  }
  __device__ __forceinline__ void st8(uint32_t o, const float (&v)[8]) const {
    st(o, make_float4(v[0], v[1], v[2], v[3]));
    st(o + plane, make_float4(v[4], v[5], v[6], v[7]));
  }
  // offset of 4 steps' entry within a stream of 2 planes per record
  __device__ __forceinline__ uint32_t half(int r) const { return (r >> 2 & 1) * plane; }
  // shared-memory offsets of the 4 positions from row r of a column
  __device__ __forceinline__ uint2 positions(bool lower, int r, int col) const {
    return ld2(record(lower, r >> 3) + index() + 16 * col + ((r & 4) << 1));
  }
};

__device__ __forceinline__ void put(float (&b)[8], float4 x, float4 y) {
  b[0] = x.x; b[1] = x.y; b[2] = x.z; b[3] = x.w; b[4] = y.x; b[5] = y.y; b[6] = y.z; b[7] = y.w;
}

// The ring: requests go round the stages in order, and so do the reads.
template <class S>
struct Ring {
  static constexpr uint32_t NT = S::kThreads;
  static constexpr uint32_t kStage = 16u * NT * kEntries;
  uint32_t smem, first, at;  // shared-memory address of res_smem; the thread's entry in stage 0 and in
                             // the next stage, bytes from there
  __device__ __forceinline__ Ring() {
    smem = static_cast<uint32_t>(__cvta_generic_to_shared(res_smem));
    first = res_ring_at(NT) + 16u * threadIdx.x;
    at = first;
  }
  // requests the parity planes and the positions of the record at `src` into the stage at `to`
  __device__ __forceinline__ void request(uint32_t to, const char* src, const uint32_t plane, bool any) const {
    if (any) {
      to += smem;
      copy(to, src);
      copy(to + 16u * NT, src + plane);
      copy(to + 32u * NT, src + 2 * plane);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  static __device__ __forceinline__ void copy(uint32_t to, const char* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
  }
  __device__ __forceinline__ void wait() const {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
  }
  __device__ __forceinline__ float4 ld(int entry) const {
    return *reinterpret_cast<const float4*>(res_smem + at + 16u * NT * entry);
  }
  __device__ __forceinline__ void advance() {
    at += kStage;
    if (at == first + kStages * kStage) at = first;
  }
  // The inputs of the 8 steps in the next stage: their places in X (w: 8 x uint16 byte offsets), the
  // LLRs s there, the parities b.
  __device__ __forceinline__ uint4 read(const char* X, float (&s)[8], float (&b)[8]) const {
    wait();
    const float4 q = ld(2);
    const uint4 w = make_uint4(__float_as_uint(q.x), __float_as_uint(q.y), __float_as_uint(q.z), __float_as_uint(q.w));
#pragma unroll
    for (int t = 0; t < 8; ++t) s[t] = lds(X, place(w, t));
    put(b, ld(0), ld(1));
    return w;
  }
  static __device__ __forceinline__ uint32_t place(const uint4& w, int t) {
    const uint32_t q = t < 2 ? w.x : t < 4 ? w.y : t < 6 ? w.z : w.w;
    return t & 1 ? q >> 16 : q & 0xffffu;
  }
};

// One SISO half-iteration of one window in the linear domain, first part: everything that reads
// other windows' positions of X.  Leaves the alpha checkpoints and the next window's alpha seed,
// and beta at the window's end in `be`; `fall` becomes the largest rescaling of the window's alpha, `least`
// (plain form) its steps' smallest weight.
template <bool STD, class W, class S>
__device__ __forceinline__ void lin_read(const ResWin& v, const Slot<S>& m, const int it, const bool lower,
                                         float (&be)[8], float& fall, float& least) {
  const uint32_t kPlane = m.plane, kRecord = 5 * m.plane;
  const char* const X = res_x<S>();
  const int tid = v.tid, G = v.guard;
  const uint32_t seed_in = m.seeds(lower, it), seed_out = m.seeds(lower, it + 1);
  float al[8];
  // ---- alpha: warm-up over the last `guard` steps of the previous window, then the window ----
  {
    const int gl = v.len >> 3;
    int j = v.nwin > 1 ? -(G >> 3) : 0;  // 8-step group; negative in the warm-up
    const int row0 = j < 0 ? v.window - G : 0, col0 = j < 0 ? v.prev : tid;
    uint32_t ck = m.ckpt(0) + 16u * tid;
    // i, src: the group that is requested next (the window's own first one follows the warm-up's last)
    Ring<S> ring;
    int i = j;
    const char* const own = m.base + m.record(lower, 0) + 16u * tid;
    const char* src = m.base + m.record(lower, row0 >> 3) + 16u * col0;
    auto request = [&](uint32_t to) {
      ring.request(to, src, kPlane, i < gl);
      src = ++i == 0 ? own : src + kRecord;
    };
#pragma unroll
    for (int st = 0; st < kStages; ++st) request(ring.at + st * Ring<S>::kStage);
    const float start = __int_as_float((v.top + 127) << 23);
    if (v.lo - G > 0) {
      float sd[8];
      m.ld8(seed_in + 16 * tid, sd);
      lin_from_log(sd, al, v.top);
    } else {
#pragma unroll
      for (int n = 0; n < 8; ++n) al[n] = n == 0 ? start : 0.0f;
    }
#pragma unroll 1
    for (; j < gl; ++j) {
      if (j == 0 && v.w == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) al[k] = k == 0 ? start : 0.0f;
      }
      float s[8], b[8];
      ring.read(X, s, b);
      const float r = rescale(al, v.top);
#pragma unroll
      for (int n = 0; n < 8; ++n) al[n] *= r;
      if (j >= 0) {
        const float o[8] = {al[0], al[4], al[1], al[5], al[2], al[6], al[3], al[7]};  // the pairs of step 0
        m.st8(ck, o);
        ck += 2 * kPlane;
        fall = fmaxf(fall, r);
      }
      request(ring.at);
      ring.advance();
      float low = 1.0f;
#pragma unroll
      for (int t = 0; t < 8; t += 2) {
        W w[2];
        weights(s[t], b[t], w[0]);
        weights(s[t + 1], b[t + 1], w[1]);
        low = least_of<STD>(low, w[0], w[1]);
        alpha_next<STD>(t, al, w[0]);
        alpha_next<STD>(t + 1, al, w[1]);
      }
      if (j >= 0) least = fminf(least, low);
    }
  }
  const int tail_at = v.k - (v.lo + v.len);  // steps of the block behind the window
  // ---- beta: warm-up over the first `guard` steps of the next window ----
  float tb[8];
  m.ld8((tail_at <= G ? m.tail(lower) : seed_in + 2 * kPlane) + 16 * tid, tb);
  const bool seed_next = v.w + 1 < v.nwin;
  if (seed_next) {  // the next window's alpha seed: alpha at hi - guard
    float sd[8];
    if (G > 0) {
      float o[8];
      m.ld8(m.ckpt((v.len - G) >> 3) + 16 * tid, o);
#pragma unroll
      for (int k = 0; k < 8; ++k) al[(k >> 1) + 4 * (k & 1)] = o[k];
    }
    log_from_lin(al, sd);
    m.st8(seed_out + 16 * v.next, sd);
  }
  lin_from_log(tb, tb, v.top);
#pragma unroll
  for (int n = 0; n < 8; ++n) be[n] = tb[n];
  if (v.nwin > 1 && G > 0) {
    Ring<S> ring;
    int j = (G >> 3) - 1, i = j;
    const char* src = m.base + m.record(lower, j) + 16u * v.next;
    auto request = [&](uint32_t to) {
      ring.request(to, src, kPlane, i >= 0);
      --i;
      src -= kRecord;
    };
#pragma unroll
    for (int st = 0; st < kStages; ++st) request(ring.at + st * Ring<S>::kStage);
#pragma unroll 1
    for (; j >= 0; --j) {
      if (8 * (j + 1) == tail_at) {
#pragma unroll
        for (int k = 0; k < 8; ++k) be[k] = tb[k];
      }
      float s[8], b[8];
      ring.read(X, s, b);
      request(ring.at);
      ring.advance();
      const float r = rescale(be, v.top);
#pragma unroll
      for (int t = 7; t >= 0; --t) {
        W w;
        weights(s[t], b[t], w);
        beta_next<STD>(t, be, w, t == 7 ? r : 1.0f);
      }
    }
    if (tail_at == 0) {
#pragma unroll
      for (int n = 0; n < 8; ++n) be[n] = tb[n];
    }
  }
}

// Second part, 8 steps at a time, last to first: alpha recomputed from its checkpoint, beta and the
// extrinsic; the previous window's beta seed is beta at lo + guard.  Replaces the LLRs of the
// window's own positions in X by the other SISO's input Ls + extrinsic, or (post) by the posterior;
// with keep_ext the extrinsics stay in the checkpoint planes too, with keep what was read (should a
// check fail).  Returns the largest |x| and the smallest mass of all paths, less what beta fell by in its
// group beyond kKept bits (0: an overflow or a NaN).
template <bool STD, class W, class S>
__device__ __forceinline__ float2 lin_write(const ResWin& v, const Slot<S>& m, const int it, const bool lower,
                                            float (&be)[8], const float scale, const bool post,
                                            const bool keep_ext, const bool keep) {
  const uint32_t kPlane = m.plane, kRecord = 5 * m.plane;
  char* const X = res_x<S>();
  const int tid = v.tid, G = v.guard;
  const uint32_t seed_out = m.seeds(lower, it + 1) + 2 * kPlane + 16 * v.prev;
  float xmax = 0.0f, smax = 0.0f, mass = 3.0e38f;  // checks
  const bool rec = v.w > 0 && G <= v.len;
  Ring<S> ring;
  int j = (v.len >> 3) - 1, i = j;
  const char* src = m.base + m.record(lower, j) + 16u * tid;
  const char* ls = src + m.sys();
  char* ck = m.base + m.ckpt(j) + 16u * tid;
  const uint32_t kept = m.kept(0) - m.ckpt(0);
  auto request = [&](uint32_t to) {
    ring.request(to, src, kPlane, i >= 0);
    --i;
    src -= kRecord;
  };
#pragma unroll
  for (int st = 0; st < kStages; ++st) request(ring.at + st * Ring<S>::kStage);
  auto ld = [](const char* p) { return *reinterpret_cast<const float4*>(p); };
  float4 ca = ld(ck), cb = ld(ck + kPlane), la = ld(ls), lb = ld(ls + kPlane);
  if (rec && v.len == G) {
    float sd[8];
    log_from_lin(be, sd);
    m.st8(seed_out, sd);
  }
#pragma unroll 1
  for (; j >= 0; --j) {
    float s[8], b[8], a[8], base[8];
    const uint4 places = ring.read(X, s, b);
    a[0] = ca.x; a[4] = ca.y; a[1] = ca.z; a[5] = ca.w;  // (the order of the checkpoints)
    a[2] = cb.x; a[6] = cb.y; a[3] = cb.z; a[7] = cb.w;
    put(base, la, lb);
    if (post) {
#pragma unroll
      for (int t = 0; t < 8; ++t) base[t] = s[t];
    }
    request(ring.at);
    ring.advance();
    char* const here = ck;
    if (W::kWide && keep) {
      *reinterpret_cast<float4*>(here + kept) = make_float4(s[0], s[1], s[2], s[3]);
      *reinterpret_cast<float4*>(here + kept + kPlane) = make_float4(s[4], s[5], s[6], s[7]);
    }
    if (j > 0) {
      ck -= 2 * kPlane;
      ls -= kRecord;
      ca = ld(ck);
      cb = ld(ck + kPlane);
      la = ld(ls);
      lb = ld(ls + kPlane);
    }
    W wt[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) weights(s[t], b[t], wt[t]);
    const float rb = rescale(be, v.top);
    // A[t]: alpha_{t+1} without its input weight (reference code) or alpha_t (TS 36.212)
    float A[8][8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      if constexpr (STD) {
#pragma unroll
        for (int n = 0; n < 8; ++n) A[t][n] = a[n];
        if (t < 7) alpha_next<STD>(t, a, wt[t]);
      } else {
        alpha_lin_at(t, a, wt[t].b, A[t]);
        if (t < 7) alpha_input(t, A[t], wt[t], a);
      }
    }
    float e[8], xl = 0.0f;
#pragma unroll
    for (int t = 7; t >= 0; --t) {
      float s1, s0;
      if constexpr (STD) {
        // sums over the branches of each input and parity
        float z[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          const int p0 = 2 * (n & 3);
          float& x0 = z[pred_input<true>(n, 0)][pred_parity(n, 0)];
          x0 = fmaf(A[t][p0], be[n], x0);
          float& x1 = z[pred_input<true>(n, 1)][pred_parity(n, 1)];
          x1 = fmaf(A[t][p0 + 1], be[n], x1);
        }
        s1 = fmaf(wt[t].b, z[1][1], z[1][0]);
        s0 = fmaf(wt[t].b, z[0][1], z[0][0]);
      } else {
        // states entered with input 1: {1, 2, 4, 7}; with input 0: {0, 3, 5, 6}
        s1 = A[t][1] * be[1];
        s0 = A[t][0] * be[0];
        s1 = fmaf(A[t][2], be[2], s1);
        s0 = fmaf(A[t][3], be[3], s0);
        s1 = fmaf(A[t][4], be[4], s1);
        s0 = fmaf(A[t][5], be[5], s0);
        s1 = fmaf(A[t][7], be[7], s1);
        s0 = fmaf(A[t][6], be[6], s0);
      }
      const float x = log_ratio(s1, s0);
      if (t & 1) xl = x;
      else xmax = max3(xmax, fabsf(x), fabsf(xl));
      smax = max3_nan(smax, s1, s0);
      // (at t = 7 beta is not rescaled yet)
      if (t == 7) mass = min_nan(mass, fminf(rb, static_cast<float>(1 << kKept)) * mass_of(wt[t], s1, s0));
      e[t] = scale * x;
      *reinterpret_cast<float*>(X + Ring<S>::place(places, t)) = base[t] + e[t];
      if (keep_ext && (t & 3) == 0)
        *reinterpret_cast<float4*>(here + (t >> 2) * kPlane) = make_float4(e[t], e[t + 1], e[t + 2], e[t + 3]);
      beta_next<STD>(t, be, wt[t], t == 7 ? rb : 1.0f);
    }
    if (rec && 8 * j == G) {
      float sd[8];
      log_from_lin(be, sd);
      m.st8(seed_out, sd);
    }
  }
  return make_float2(xmax, smax < 0x1p126f && mass > 0.0f ? mass : 0.0f);
}

// A half-iteration of the CTA's blocks in the linear domain; `run`: this thread's window takes part.
// Returns the bits by which its block passed the checks (negative: it did not), and whether it ran: in the
// plain form a block with a weight below 2^-126 is left as it was (below 0).
template <bool STD, class W, class S>
__device__ __noinline__ float2 lin_half(bool run, const int half, const float scale, const bool post,
                                        const bool keep_ext, const bool keep) {
  const ResWin v = res_win<S>();
  const Slot<S> m;
  const bool lower = half & 1;
  float be[8], fall = 1.0f, least = 1.0f;
  if (run) lin_read<STD, W, S>(v, m, half >> 1, lower, be, fall, least);
  __syncthreads();  // every window has read X (and left its seeds and checkpoints)
  float ran = 1.0f;
  if constexpr (!W::kWide) {
    res_word<S>(kWordMass)[threadIdx.x] = 0x3f800000;
    __syncthreads();
    if (run) atomicMin(res_word<S>(kWordMass) + v.lane0, __float_as_int(least));
    __syncthreads();
    if (__int_as_float(res_word<S>(kWordMass)[v.lane0]) < 0x1p-126f) {
      ran = -1.0f;
      run = false;
    }
    __syncthreads();  // (the ring is in use again)
  }
  float2 c = make_float2(0.0f, 0.0f);
  if (run) c = lin_write<STD, W, S>(v, m, half >> 1, lower, be, scale, post, keep_ext, keep);
  __syncthreads();
  res_word<S>(kWordExt)[threadIdx.x] = 0;
  res_word<S>(kWordMass)[threadIdx.x] = 0x7f000000;
  res_word<S>(kWordFall)[threadIdx.x] = 0x3f800000;
  __syncthreads();
  if (run) {
    atomicMax(res_word<S>(kWordExt) + v.lane0, __float_as_int(c.x));
    atomicMin(res_word<S>(kWordMass) + v.lane0, __float_as_int(c.y));
    atomicMax(res_word<S>(kWordFall) + v.lane0, __float_as_int(fall));
  }
  __syncthreads();
  const auto word = [&](int i) { return __int_as_float(res_word<S>(i)[v.lane0]); };
  const float lost = !STD && !W::kWide ? word(kWordPar) : 0.0f;  // by the plain form's beta
  return make_float2(lg2(word(kWordMass)) - word(kWordExt) - (static_cast<float>(v.top) - kLost) - lost -
                         fmaxf(lg2(word(kWordFall)) - static_cast<float>(kKept), 0.0f),
                     ran);
}

// The extrinsics in the checkpoint planes into X: added to Ls (the other SISO's input), or (post)
// to what stands there (the posterior).
template <class S>
__device__ __noinline__ void put_extrinsics(const bool lower, const bool post) {
  const ResWin v = res_win<S>();
  const Slot<S> m;
  char* const X = res_x<S>();
  // 32 steps at a time, all loads before any use (rows behind the window repeat its last ones)
  constexpr int kPart = 4;
#pragma unroll 1
  for (int r0 = 0; r0 < v.len; r0 += 8 * kPart) {
    float e[kPart][8], l[kPart][8];
    uint4 q[kPart];
#pragma unroll
    for (int i = 0; i < kPart; ++i) {
      const int g = min(r0 + 8 * i, v.len - 8) >> 3;
      m.ld8(m.ckpt(g) + 16 * v.tid, e[i]);
      m.ld8(m.record(lower, g) + m.sys() + 16 * v.tid, l[i]);
      q[i] = *reinterpret_cast<const uint4*>(m.base + m.record(lower, g) + m.index() + 16 * v.tid);
    }
#pragma unroll
    for (int i = 0; i < kPart; ++i) {
      if (r0 + 8 * i >= v.len) break;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        float* d = reinterpret_cast<float*>(X + Ring<S>::place(q[i], t));
        *d = (post ? *d : l[i][t]) + e[i][t];
      }
    }
  }
}

// X of this thread's window as the half-iteration that failed had it, in natural units.
template <class S>
__device__ __noinline__ void res_restore(const bool lower) {
  const ResWin v = res_win<S>();
  const Slot<S> m;
  char* const X = res_x<S>();
#pragma unroll 2
  for (int g = 0; g < v.len >> 3; ++g) {
    float s[8];
    m.ld8(m.kept(g) + 16 * v.tid, s);
    const uint4 q = *reinterpret_cast<const uint4*>(m.base + m.record(lower, g) + m.index() + 16 * v.tid);
#pragma unroll
    for (int t = 0; t < 8; ++t) *reinterpret_cast<float*>(X + Ring<S>::place(q, t)) = kLn2 * s[t];
  }
}

// A warp's windows by block: calls f(lane of the block's first window in this warp, steps) for each
// block (its windows in a warp are consecutive lanes, their steps consecutive in every stream).
template <class F>
__device__ __forceinline__ void res_for_blocks(const ResWin& v, F f) {
  const int lane = threadIdx.x & 31;
  unsigned first = __ballot_sync(0xffffffffu, v.len > 0 && (v.w == 0 || lane == 0));
  while (first) {
    const int l = __ffs(first) - 1;
    first &= first - 1;
    // up to the block's end, or to the end of the warp's last lane
    const int k = __shfl_sync(0xffffffffu, v.k, l), lo = __shfl_sync(0xffffffffu, v.lo, l);
    f(l, min(k - lo, (32 - l) * __shfl_sync(0xffffffffu, v.window, l)), __shfl_sync(0xffffffffu, v.window, l));
  }
}

// Copies the windows' rows (entries of SIZE bytes; `src`: this lane's window) to stage + thread *
// pitch, each warp its own with consecutive 16-byte pieces per lane, and waits for them.
template <int SIZE>
__device__ __forceinline__ void res_stage_rows(const ResWin& v, const void* src, char* stage, int pitch) {
  const int lane = threadIdx.x & 31;
  const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(stage)) + (threadIdx.x & ~31) * pitch;
  constexpr int kPiece = 16 / SIZE;
  res_for_blocks(v, [&](int l, int steps, int window) {
    const char* p = reinterpret_cast<const char*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(src), l));
    const uint32_t inv = 0xffffffffu / static_cast<uint32_t>(window) + 1u;
#pragma unroll 4
    for (int q = kPiece * lane; q < steps; q += kPiece * 32) {
      const int w = __umulhi(q, inv);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + (l + w) * pitch + (q - w * window) * SIZE),
                   "l"(p + q * SIZE)
                   : "memory");
    }
  });
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
}

// The inputs of a task, in base-2 units with parity weights for the linear pass: the streams' planes, X = the systematic LLRs (the first input of
// the upper SISO), the interleaved positions, the tail betas; seeds zero if the block starts here (`start`; one
// that goes on keeps the seeds of the half-iterations before).
// Each warp stages its windows' rows through shared memory (where X and the ring will be; a row
// pitch of an odd number of 16-byte words keeps both sides free of bank conflicts).
template <bool STD, class S>
__device__ __noinline__ void res_inputs(const ResCb* cb, const float* llr, const uint16_t* perm,
                                        const bool linear, const bool start) {
  const Slot<S> m;
  const float unit = linear ? kLog2e : 1.0f;
  const int tid = threadIdx.x;
  const bool mine = cb != nullptr;
  const ResWin v = res_win<S>();
  char* const X = res_x<S>();
  char* const stage = res_smem + res_ring_at(S::kThreads);
  const int W = res_cta().max_window;
  const float* const d0 = mine ? llr + cb->llr : nullptr;
  __syncthreads();
  {  // positions: rows of uint16
    const int pitch = 2 * W + 16;
    // a row starts at any multiple of 8 entries: 16-byte aligned
    res_stage_rows<2>(v, mine ? perm + cb->tab + v.lo : nullptr, stage, pitch);
    if (mine) {
      const uint32_t inv = 0xffffffffu / static_cast<uint32_t>(v.window) + 1u;
      const char* row = stage + tid * pitch;
#pragma unroll 2
      for (int r = 0; r < v.window; r += 8) {
        uint32_t o[8];
        if (r < v.len) {
          const uint4 q = *reinterpret_cast<const uint4*>(row + 2 * r);
          const uint32_t n[8] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16,
                                 q.z & 0xffffu, q.z >> 16, q.w & 0xffffu, q.w >> 16};
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const uint32_t w = __umulhi(n[t], inv);
            o[t] = (n[t] - w * v.window) * v.xs4 + 4u * (v.lane0 + w);
          }
        } else {  // behind the block's last step: any place
#pragma unroll
          for (int t = 0; t < 8; ++t) o[t] = 4u * tid;
        }
        *reinterpret_cast<uint4*>(m.base + m.record(true, r >> 3) + m.index() + 16u * tid) =
            make_uint4(o[0] | o[1] << 16, o[2] | o[3] << 16, o[4] | o[5] << 16, o[6] | o[7] << 16);
        const uint32_t own = r * v.xs4 + 4u * tid, two = own | own << 16, step = v.xs4 | v.xs4 << 16;
        *reinterpret_cast<uint4*>(m.base + m.record(false, r >> 3) + m.index() + 16u * tid) =
            make_uint4(two + (v.xs4 << 16), two + 2 * step + (v.xs4 << 16), two + 4 * step + (v.xs4 << 16),
                       two + 6 * step + (v.xs4 << 16));
      }
    }
    __syncwarp();
  }
  const int pitch = 4 * W + 16;
#pragma unroll 1
  for (int st = 0; st < 3; ++st) {  // parity 1, parity 2, systematic
    const int which = st == 2 ? 0 : st + 1;
    if (S::kThreads > 32) __syncthreads();  // (pitches differ: a row may lie in another warp's part)
    res_stage_rows<4>(v, mine ? d0 + which * (v.k + 4) + v.lo : nullptr, stage, pitch);
    if (mine) {
      const char* row = stage + tid * pitch;
      float most = 0.0f;
      const bool exp_now = linear && which != 0;
#pragma unroll 4
      for (int r = 0; r < v.window; r += 4) {
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < v.len) x = *reinterpret_cast<const float4*>(row + 4 * r);
        x = make_float4(unit * x.x, unit * x.y, unit * x.z, unit * x.w);
        const auto size = [](float y) { return y < -kVoid ? 0.0f : fabsf(y); };
        most = max3(max3(most, size(x.x), size(x.y)), size(x.z), size(x.w));
        if (exp_now) x = make_float4(ex2(x.x), ex2(x.y), ex2(x.z), ex2(x.w));
        m.st(m.record(which == 2, r >> 3) + (which == 0 ? m.sys() : 0) + m.half(r) + 16u * tid, x);
      }
      if (which != 0) atomicMax(res_word<S>(kWordPar) + v.lane0, __float_as_int(most));
    }
    __syncwarp();
  }
  __syncthreads();
  if (mine) {
    // 32 steps at a time, all loads before any store
#pragma unroll 1
    for (int r0 = 0; r0 < v.len; r0 += 32) {
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = min(r0 + 4 * i, v.len - 4);
        x[i] = m.ld(m.record(false, r >> 3) + m.sys() + m.half(r) + 16 * tid);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (r0 + 4 * i >= v.len) break;
        char* d = X + (r0 + 4 * i) * v.xs4 + 4 * tid;
        *reinterpret_cast<float*>(d) = x[i].x;
        *reinterpret_cast<float*>(d + v.xs4) = x[i].y;
        *reinterpret_cast<float*>(d + 2 * v.xs4) = x[i].z;
        *reinterpret_cast<float*>(d + 3 * v.xs4) = x[i].w;
      }
    }
  }
  __syncthreads();
  if (!mine) return;
#pragma unroll 1
  for (int r0 = 0; r0 < v.window; r0 += 32) {
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      q[i] = *reinterpret_cast<const uint4*>(
          m.base + m.record(true, min(r0 + 8 * i, v.window - 8) >> 3) + m.index() + 16u * tid);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (r0 + 8 * i >= v.window) break;
      const uint32_t at = m.record(true, (r0 >> 3) + i) + m.sys() + 16u * tid;
      m.st(at, make_float4(lds(X, q[i].x & 0xffffu), lds(X, q[i].x >> 16), lds(X, q[i].y & 0xffffu),
                           lds(X, q[i].y >> 16)));
      m.st(at + m.plane, make_float4(lds(X, q[i].z & 0xffffu), lds(X, q[i].z >> 16),
                                      lds(X, q[i].w & 0xffffu), lds(X, q[i].w >> 16)));
    }
  }
  const uint32_t sd = m.seeds(false, 0) + 16u * tid;
#pragma unroll 1
  for (int i = 0; start && i < 16; ++i) m.st(sd + i * m.plane, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
  if (v.k - (v.lo + v.len) <= v.guard) {
#pragma unroll
    for (int lower = 0; lower < 2; ++lower) {
      float ts[3], tp[3], tb[8];
      tail_llrs<STD>(lower, d0, v.k, ts, tp);
      tail_beta<STD>(tb, ts, tp);
      m.st8(m.tail(lower) + 16u * tid, tb);
    }
  }
}

// This window's part of its block's CRC24B syndrome of the hard decisions [filler, K)
// (lte_turbo.cpp:792-804): the window's bits modulo g 4 at a time, times x^(steps behind it).
template <class S>
__device__ __noinline__ void res_crc(const uint32_t* xpow, const int filler) {
  const ResWin v = res_win<S>();
  const char* const X = res_x<S>();
  const uint32_t* const tab = res_cta().crc_tab;
  uint32_t c = 0, off = 4u * v.tid;
#pragma unroll 4
  for (int r = 0; r < v.len; r += 8) {
    uint32_t byte = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t, off += v.xs4) {
      const bool bit = lds(X, off) >= 0.0f && v.lo + r + t >= filler;
      byte = 2 * byte + (bit ? 1u : 0u);
    }
    c = ((c << 4) & 0xffffffu) ^ tab[c >> 20] ^ (byte >> 4);
    c = ((c << 4) & 0xffffffu) ^ tab[c >> 20] ^ (byte & 15u);
  }
  uint32_t z = 0;
  const uint32_t* xp = xpow + (v.k - (v.lo + v.len));
#pragma unroll
  for (int b = 0; b < 24; ++b) z ^= (c >> b) & 1u ? __ldg(xp + b) : 0u;
  atomicXor(reinterpret_cast<uint32_t*>(res_word<S>(kWordSyn)) + v.lane0, z);
}

// The posteriors in X, times `unit`, of the windows whose lane has a `dst` to there, each warp its own
// windows.
template <class S>
__device__ __noinline__ void res_outputs(float* dst, const float unit) {
  const ResWin v = res_win<S>();
  const int lane = threadIdx.x & 31;
  const char* const X = res_x<S>() + 4 * (v.tid - lane);
  res_for_blocks(v, [&](int l, int steps, int window) {
    float* const p = reinterpret_cast<float*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(dst), l));
    if (p == nullptr) return;
    const uint32_t inv = 0xffffffffu / static_cast<uint32_t>(window) + 1u;
#pragma unroll 8
    for (int q = lane; q < steps; q += 32) {
      const int w = __umulhi(q, inv);
      p[q] = unit * lds(X, (q - w * window) * v.xs4 + 4u * (l + w));
    }
  });
}

// ---- (m, s) pass: blocks whose metrics left float's range, in the form of siso.cuh, with
// X and the planes in natural units ----
template <bool LOWER, class S>
struct SlotAccess {
  ResWin v;
  Slot<S> m;
  uint32_t seed_in, seed_out;
  float factor;
  const float* d0;
  __device__ __forceinline__ int guard() const { return v.guard; }
  __device__ __forceinline__ float scale() const { return factor; }
  // 4 steps from q (of the block), which may lie in a neighbouring window
  __device__ __forceinline__ Raw4 raw4(int q) const {
    int row = q - v.lo, col = v.tid;
    if (row < 0) {
      row += v.window;
      --col;
    } else if (row >= v.window) {
      row -= v.window;
      ++col;
    }
    const char* const X = res_x<S>();
    const uint2 w = m.positions(LOWER, row, col);
    return Raw4{make_float4(lds(X, w.x & 0xffffu), lds(X, w.x >> 16), lds(X, w.y & 0xffffu), lds(X, w.y >> 16)),
                make_float4(0.0f, 0.0f, 0.0f, 0.0f),
                m.ld(m.record(LOWER, row >> 3) + m.half(row) + 16 * col)};
  }
  __device__ __forceinline__ Raw8 raw8(int q) const { return Raw8{raw4(q), raw4(q + 4)}; }
  __device__ __forceinline__ void load_seed(bool beta, float (&x)[8]) const {
    m.ld8(seed_in + (beta ? 2 * m.plane : 0) + 16 * v.tid, x);
  }
  __device__ __forceinline__ void store_seed(bool beta, const float (&x)[8]) const {
    m.st8(seed_out + (beta ? 2 * m.plane + 16 * v.prev : 16 * v.next), x);
  }
  __device__ __forceinline__ uint2 targets(int) const { return make_uint2(0, 0); }
  __device__ __forceinline__ void put(int q, int, float e, float) const {
    const int row = q - v.lo;
    *reinterpret_cast<float*>(m.base + m.ckpt(row >> 3) + m.half(row) + 16 * v.tid + 4 * (row & 3)) = e;
  }
};

// A half-iteration of this thread's window: reads X, leaves the extrinsics in the checkpoint planes.
template <bool LOWER, bool STD, class S>
__device__ __noinline__ void log_half(const float* d0, const int it, const float scale) {
  SlotAccess<LOWER, S> io;
  io.v = res_win<S>();
  io.seed_in = io.m.seeds(LOWER, it);
  io.seed_out = io.m.seeds(LOWER, it + 1);
  io.factor = scale;
  io.d0 = d0;
  DevCb cb{};
  cb.k = io.v.k;
  cb.nwin = io.v.nwin;
  cb.window = io.v.window;
  const int pitch = io.m.plane / 16;
  const CkptStrided ck{reinterpret_cast<float4*>(io.m.base) + 12 * io.m.rows8 * pitch, pitch, io.v.tid};
  siso_window<kSub, LOWER, STD, false>(cb, io.v.w, io, ck);
}

// The two-factor form is called through a pointer (volatile: the compiler may not see through it): as a
// direct call of the kernel it takes registers from the plain form, which needs all of them (12 to 28 bytes
// of spills in its loops, 4096 blocks of K = 6144 2.82 ms instead of 2.67).
using LinHalf = float2 (*)(bool, int, float, bool, bool, bool);
template <bool STD, class S>
__device__ volatile LinHalf wide_half = lin_half<STD, WideWeights, S>;

template <bool STD, class S>
__global__ void __launch_bounds__(S::kThreads, 256 / S::kThreads) resident_kernel(const __grid_constant__ ResArgs p) {
  const int tid = threadIdx.x;
  ResCta& cta = res_cta();
  for (int task = blockIdx.x; task < p.n_tasks;) {
    if (task == p.stall_task && tid == 0) {  // testing hook: a wait that runs out
      const uint64_t t0 = global_ns();
      while (load_acquire(p.never) == 0) {
        if (global_ns() - t0 > kWaitLimitNs) {
          atomicExch(p.error, 1);
          break;
        }
        __nanosleep(256);
      }
    }
    const int first = p.task_first[task], last = p.task_first[task + 1];
    const ResCb* cb = nullptr;  // this thread's block
    int lane0 = 0, lanes = 0, max_window = 0;
    ushort4 win = make_ushort4(0, 0, 0, 0);
    for (int c = first; c < last; ++c) {
      const ResCb& o = p.cbs[c];
      const int l0 = o.lane0, n = o.nwin;
      if (tid >= l0 && tid < l0 + n) {
        cb = &o;
        lane0 = l0;
        win = make_ushort4(o.k, o.window, n, l0);
      }
      lanes = l0 + n;
      max_window = max(max_window, o.window);
    }
    const bool mine = cb != nullptr;
    res_word<S>(kWordPar)[tid] = 0;
    if (tid == 0) {
      cta.slot = reinterpret_cast<char*>(p.scratch + p.slot * blockIdx.x);
      cta.guard = p.guard;
      cta.rows8 = max_window / 8;
      cta.plane = 16u * lanes;
      cta.xs4 = 4u * res_pitch(lanes);
      cta.max_window = max_window;
    }
    if (tid < 16) cta.crc_tab[tid] = __ldg(p.xpow + kXpowSize + tid);
    __syncthreads();
    res_window<S>()[tid] = win;  // read by this thread alone
    bool passed = false;
    int used = p.max_iterations;

    // Three passes: all blocks in the plain linear form, as far as it goes; what is left in the two-factor
    // form, from X as it stands; and what that one leaves in the (m, s) form.  `done_in` is the pass that a
    // block ends in, `from` the half-iteration where that pass takes over.
    int done_in = kPlain, from = 0;
    float margin = 1000.0f;  // of the block's checks in the last half-iteration
#pragma unroll 1
    for (int pass = kPlain; pass <= kLog && p.max_iterations > 0; ++pass) {
      bool run = mine && done_in == pass;
      if (pass != kPlain && !__syncthreads_or(run)) continue;
      const bool taken = run;
      if (pass != kWide) {
        res_inputs<STD, S>(cb, p.llr, p.perm, pass == kPlain, from == 0);
        __syncthreads();
      }
      if (pass == kLog) {
        if (run && from > 0) res_restore<S>(from & 1);
        __syncthreads();
      }
      if (pass == kPlain) {
        const bool outside = run && __int_as_float(res_word<S>(kWordPar)[lane0]) > kMaxParity;
        if (outside) {
          done_in = kLog;
          run = false;
        }
      }
#pragma unroll 1
      for (int half = 0; half < 2 * p.max_iterations; ++half) {
        const int it = half >> 1;
        const bool lower = half & 1, last_half = half + 1 == 2 * p.max_iterations;
        const bool post_now = lower && (p.early_stop || last_half);
        const float scale = __ldg(p.scale + half);
        if (pass == kPlain) {
          if (run && margin < kNearPlain) {
            done_in = kWide;
            from = half;
            run = false;
          }
          if (!__syncthreads_or(run)) break;
          const float2 c = lin_half<STD, Weights, S>(run, half, scale, post_now, lower && p.early_stop, false);
          if (run && c.y < 0.0f) {
            done_in = kWide;
            from = half;
            run = false;
          } else if (run) {
            margin = c.x;
            if (!(margin >= 0.0f)) {
              done_in = kLog;
              run = false;
            }
          }
        } else if (pass == kWide) {
          const bool now = run && half >= from;
          if (!__syncthreads_or(now)) continue;
          const bool keep = margin < kNear;
          const float2 c = wide_half<STD, S>(now, half, scale, post_now, lower && p.early_stop, keep);
          if (now) {
            margin = c.x;
            if (!(margin >= 0.0f)) {
              done_in = kLog;
              from = keep ? half : 0;
              run = false;
            }
          }
        } else {
          if (run && half >= from) {
            const float* d0 = p.llr + cb->llr;
            if (lower) log_half<true, STD, S>(d0, it, scale);
            else log_half<false, STD, S>(d0, it, scale);
          }
          __syncthreads();
          if (run && half >= from) put_extrinsics<S>(lower, post_now);
        }
        __syncthreads();
        if (post_now && p.early_stop) {
          res_word<S>(kWordSyn)[tid] = 0;
          __syncthreads();
          if (run && half >= from) res_crc<S>(p.xpow, cb->filler);
          __syncthreads();
          if (run && half >= from) {
            used = it + 1;
            passed = res_word<S>(kWordSyn)[lane0] == 0;
            // X goes from the posterior to the next iteration's input
            if (!passed && !last_half) put_extrinsics<S>(true, false);
            run = !passed;
          }
          if (!__syncthreads_or(run)) break;
        }
      }
      const bool write = taken && done_in == pass;
      res_outputs<S>(write ? p.post + cb->out + (tid - lane0) * cb->window : nullptr,
                      pass != kLog ? kLn2 : 1.0f);
      __syncthreads();
    }
    if (mine && tid == lane0) {
      p.crc_ok[cb->idx] = passed ? 1 : 0;
      p.iters[cb->idx] = static_cast<uint32_t>(used);
    }
    if (p.n_tasks <= static_cast<int>(gridDim.x)) return;
    __syncthreads();
    if (tid == 0) cta.next_task = static_cast<int>(gridDim.x) + atomicAdd(p.queue, 1);
    __syncthreads();
    task = cta.next_task;
    __syncthreads();
  }
}

}  // namespace
}  // namespace tcb
