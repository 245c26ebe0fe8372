// decode_kernels.cuh -- the kernels of one plain-schedule decode (per half-iteration SISO
// launches, set-up, CRC24B early stop), shared by the decoder object (decoder.cu) and the
// allocation-free entry point (noalloc.cu).  Each including translation unit gets its own
// internal-linkage instances.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "decoder.hpp"
#include "siso.cuh"

namespace tcb {
namespace {

constexpr int kThreads = 64;  // threads (windows) per block of the plain SISO kernel
constexpr int kMinBlocks = 8;  // 16 warps per SM: at most 128 registers per thread

// KIND: 0 = upper SISO, 1 = lower SISO, 2 = lower SISO that also writes the posterior;
// STD: the TS 36.212 code instead of the reference's; TAPE: the alpha checkpoints cover
// the warm-up too, plane (q - a_lo) / S of the slab for step q, and stay for the adjoint (a slab of
// (window + guard) / S + 1 planes).  The checkpoint slab holds planes of n_win float4 pairs (windows interleaved).
template <int S, int KIND, bool STD = false, bool TAPE = false>
__global__ void __launch_bounds__(kThreads, kMinBlocks) siso_plain_kernel(const DevCb* __restrict__ cbs,
                                                              const int32_t* __restrict__ win_cb,
                                                              int n_win, SisoIo io,
                                                              const uint8_t* __restrict__ done,
                                                              float4* ckpt) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_win) return;
  const int c = win_cb[g];
  if (done != nullptr && done[c]) return;
  const DevCb cb = cbs[c];
  const int w = g - cb.win0;
  CkptStrided ck{ckpt, n_win, g};
  if (TAPE)  // plane 0 is alpha at a_lo
    ck.p += static_cast<int64_t>(2 * (min(w * cb.window, io.guard) / S)) * n_win;
  siso_window<S, KIND != 0, STD, TAPE>(cb, w, GlobalAccess<KIND != 0, KIND == 2>(io, cb, g), ck);
}

// sys_i[i] = d0[Pi(i)]; E2 = 0 (first a-priori).  One CTA per code block: d0 is read into shared
// memory with coalesced loads, then the interleaved copy is gathered from there, so that every
// global access walks its array in order (a direct gather would read one 32-byte sector per
// 4-byte element).
constexpr int kGatherThreads = 512;
constexpr int kMaxBlockK = 6144;
__global__ void __launch_bounds__(kGatherThreads) setup_kernel(const DevCb* __restrict__ cbs,
                                                               int n_cb,
                                                               const float* __restrict__ llr,
                                                               const uint16_t* __restrict__ perm,
                                                               float* __restrict__ sys_i,
                                                               float* __restrict__ e2) {
  __shared__ float d0[kMaxBlockK];
  for (int c = blockIdx.x; c < n_cb; c += gridDim.x) {
    const DevCb cb = cbs[c];
    const float* src = llr + cb.llr;
    for (int p = threadIdx.x; p < cb.k; p += kGatherThreads) d0[p] = __ldg(src + p);
    __syncthreads();
    const uint16_t* pi = perm + cb.tab;
    for (int p = threadIdx.x; p < cb.k; p += kGatherThreads) {
      sys_i[cb.work + p] = d0[pi[p]];
      e2[cb.work + p] = 0.0f;
    }
    __syncthreads();  // d0 is reused by the next code block
  }
}

inline void launch_setup(const DevCb* cbs, int n_cb, const float* llr, const uint16_t* perm,
                         float* sys_i, float* e2, cudaStream_t st) {
  if (n_cb <= 0) return;
  const unsigned grid = static_cast<unsigned>(n_cb < (1 << 20) ? n_cb : (1 << 20));
  setup_kernel<<<grid, kGatherThreads, 0, st>>>(cbs, n_cb, llr, perm, sys_i, e2);
}

// CRC24B early stop (lte_turbo.cpp:792-804): hard decisions (>= 0 -> 1) of bits
// [filler, K) must form a codeword of the reference's CRC24B generator, i.e. the XOR of
// x^(N-1-i) mod g over the set bits i must be zero.  One warp per code block.
__global__ void crc_stop_kernel(const DevCb* __restrict__ cbs, int n_cb,
                                const float* __restrict__ post, const uint32_t* __restrict__ xpow,
                                uint8_t* __restrict__ done, uint32_t* __restrict__ iters, int it) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n_cb || done[warp]) return;
  const DevCb cb = cbs[warp];
  const int n = cb.k - cb.filler;
  const float* p = post + cb.out + cb.filler;
  uint32_t syn = 0;
  for (int i = lane; i < n; i += 32)
    if (p[i] >= 0.0f) syn ^= xpow[n - 1 - i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) syn ^= __shfl_xor_sync(0xffffffffu, syn, o);
  if (lane == 0) {
    iters[warp] = static_cast<uint32_t>(it + 1);
    if (syn == 0) done[warp] = 1;
  }
}

__global__ void init_flags_kernel(int n_cb, uint8_t* __restrict__ done, uint32_t* __restrict__ iters,
                                  uint32_t max_iterations) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_cb) {
    done[i] = 0;
    iters[i] = max_iterations;  // early stop lowers it
  }
}

__global__ void finish_kernel(int n_cb, const uint8_t* __restrict__ done, uint8_t* crc_ok,
                              int early_stop) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_cb) crc_ok[i] = early_stop ? done[i] : 0;
}

}  // namespace
}  // namespace tcb
