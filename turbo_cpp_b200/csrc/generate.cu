// generate.cu -- test-vector generation on the device: seeded information bits with CRC24B,
// the turbo encoder, the rate matcher and the BPSK/AWGN channel.  The bits, encoded streams and
// rate-matched bits are bit-identical to the host codec (lte_codec.cpp: random_bits,
// crc_append, turbo_encode, rate_match, i.e. the reference's turbo_encode_code_block
// lte_turbo.cpp:624-688 and puncture_and_collect :250-278); the channel uses the same
// counter-based draws as the host's awgn_llr, so the LLRs equal the host's up to the last bit
// of CUDA's double log/cos against the host C library's.
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <vector>

#include "circular_buffer.cuh"
#include "decoder.hpp"
#include "lte_codec.hpp"

namespace tcb {
namespace {

void ok(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw CudaError(std::string(what) + ": " + cudaGetErrorString(e));
}

// SplitMix64 finaliser (the host generator's mixing function)
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
uint64_t host_mix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

struct GenBlock {
  int32_t k, filler;
  int64_t bits;     // offset of the K information bits
  int64_t llr;      // offset of the 3(K+4) LLRs (or encoded bits)
  uint64_t seed;    // per-block stream seed
  double sigma, scale;  // channel: noise deviation, LLR scale 2 / sigma^2
};

constexpr int kGenThreads = 256;

// One CTA per block: bits[i] = top bit of mix64(key + i), the filler zeroed, and with crc24b
// the last 24 bits replaced by the CRC24B of bits [filler, K-24): the remainder is the XOR of
// x^(n-1-i) mod g over the set payload bits i (n = K - filler, table xpow), whose coefficient
// of x^(23-j) is CRC bit j -- the codeword the decoder's syndrome check accepts.
__global__ void __launch_bounds__(kGenThreads) gen_bits_kernel(const GenBlock* __restrict__ blocks,
                                                              int crc24b,
                                                              const uint32_t* __restrict__ xpow,
                                                              uint8_t* __restrict__ bits) {
  __shared__ uint32_t part[kGenThreads / 32];
  const GenBlock b = blocks[blockIdx.x];
  const uint64_t key = mix64(b.seed ^ 0x6a09e667f3bcc909ull);
  const int n = b.k - b.filler;
  const int pay_end = crc24b ? b.k - 24 : b.k;
  uint8_t* out = bits + b.bits;
  uint32_t r = 0;
  for (int i = threadIdx.x; i < b.k; i += blockDim.x) {
    uint8_t v = static_cast<uint8_t>(mix64(key + static_cast<uint64_t>(i)) >> 63);
    if (i < b.filler) v = 0;
    if (i < pay_end) {
      out[i] = v;
      if (crc24b && v) r ^= xpow[n - 1 - (i - b.filler)];
    }
  }
  if (!crc24b) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r ^= __shfl_xor_sync(0xffffffffu, r, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x < 24) {
    uint32_t x = 0;
    for (int w = 0; w < kGenThreads / 32; ++w) x ^= part[w];
    out[b.k - 24 + threadIdx.x] = static_cast<uint8_t>((x >> (23 - threadIdx.x)) & 1u);
  }
}

__device__ __forceinline__ uint8_t rsc_step(uint8_t& s, uint8_t u) {
  const uint8_t s0 = s & 1u, s1 = (s >> 1) & 1u, s2 = (s >> 2) & 1u;
  const uint8_t fb = u ^ s1 ^ s2;  // the reference's feedback u^s1^s2 (lte_turbo.cpp:337)
  s = static_cast<uint8_t>((fb << 2) | (s2 << 1) | s1);
  return fb ^ s0 ^ s2;
}

// One CTA per block, 32 steps per thread: warps 0-5 the upper encoder (natural order), 6-11 the lower
// (QPP order).  With fb the feedback bits (rsc_step), fb = u / (1 + D + D^2) = u (1 + D) / (1 + D^3)
// over GF(2): a word of 32 steps from state zero is a stride-3 prefix XOR, and what the state before it
// adds repeats every 3 steps.  The states at the words' ends are 2 bits (the last two feedback bits)
// that a word maps by B (B^3 = 1), so that an XOR scan of B^-(j+1) z_j gives every word its state.
// Bound by latency, a barrier between each of five short phases; 4096 mixed blocks: 54 us, 842 us with
// one thread stepping through each encoder bit by bit.
constexpr int kEncWords = 192;  // words of the largest block
constexpr int kEncThreads = 2 * kEncWords;

// B^n x for the 2-bit state x = fb_-1 | fb_-2 << 1: B maps (fb_-1, fb_-2) to (fb_-2, fb_-1 ^ fb_-2)
__device__ __forceinline__ uint32_t state_after(uint32_t x, int n) {
  const uint32_t p1 = x & 1u, p2 = x >> 1, both = p1 ^ p2;
  return n == 0 ? x : n == 1 ? (p2 | both << 1) : (both | p1 << 1);
}
// 4 bits as 4 bytes
__device__ __forceinline__ uint32_t spread4(uint32_t v) { return ((v & 15u) * 0x00204081u) & 0x01010101u; }

__global__ void __launch_bounds__(kEncThreads) encode_kernel(const GenBlock* __restrict__ blocks,
                                                             const uint16_t* __restrict__ perm,
                                                             const int32_t* __restrict__ tab,
                                                             const uint8_t* __restrict__ bits,
                                                             uint8_t* __restrict__ d012) {
  __shared__ uint32_t u[2][kEncWords];      // inputs of the two encoders
  __shared__ uint32_t f[2][kEncWords + 1];  // feedback words, f[.][0] = 0
  __shared__ uint32_t out[3][kEncWords];    // d0, d1, d2
  __shared__ uint32_t sums[2][kEncWords / 32];
  const GenBlock b = blocks[blockIdx.x];
  const int K = b.k, words = (K + 31) / 32;
  const int tid = threadIdx.x, lane = tid & 31;
  const uint8_t* cb = bits + b.bits;
  // inputs, a word per warp and step
  for (int i = tid; i < words * 32; i += kEncThreads) {
    const uint32_t w = __ballot_sync(0xffffffffu, i < K && (cb[i] & 1u));
    if (lane == 0) u[0][i >> 5] = w;
  }
  __syncthreads();
  const uint16_t* pm = perm + tab[blockIdx.x];
  for (int i = tid; i < words * 32; i += kEncThreads) {
    const int n = i < K ? pm[i] : 0;
    const uint32_t w = __ballot_sync(0xffffffffu, i < K && (u[0][n >> 5] >> (n & 31) & 1u));
    if (lane == 0) u[1][i >> 5] = w;
  }
  __syncthreads();
  const int enc = tid >= kEncWords, j = tid - enc * kEncWords;
  uint32_t z = 0, y = 0;
  if (j < words) {
    z = u[enc][j];
    z ^= z << 1;
    z ^= z << 3;
    z ^= z << 6;
    z ^= z << 12;
    z ^= z << 24;
    y = state_after((z >> 31) | (z >> 30 & 1u) << 1, 2 * (j + 1) % 3);
  }
  uint32_t x = y;  // inclusive scan
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x ^= v;
  }
  if (lane == 31) sums[enc][j >> 5] = x;
  __syncthreads();
  uint32_t st = x ^ y;
  for (int w = 0; w < j >> 5; ++w) st ^= sums[enc][w];
  st = state_after(st, j % 3);
  const uint32_t p1 = st & 1u, p2 = st >> 1;
  z ^= (p1 ^ p2 ? 0x49249249u : 0u) ^ (p2 ? 0x92492492u : 0u) ^ (p1 ? 0x24924924u : 0u);
  if (j < words) f[enc][j + 1] = z;
  if (j == 0) f[enc][0] = 0;
  __syncthreads();
  if (j < words) {
    const uint32_t before = f[enc][j];
    const uint32_t p = z ^ (z << 1 | before >> 31) ^ (z << 3 | before >> 29);
    if (enc == 0) {
      const int nulls = b.filler - 32 * j;  // filler bits are sent as 0 in d0 and d1
      const uint32_t keep = nulls <= 0 ? ~0u : nulls >= 32 ? 0u : ~0u << nulls;
      out[0][j] = u[0][j] & keep;
      out[1][j] = p & keep;
    } else {
      out[2][j] = p;
    }
  }
  __syncthreads();
  uint8_t* d0 = d012 + b.llr;
  uint8_t* d1 = d0 + (K + 4);
  uint8_t* d2 = d1 + (K + 4);
  const bool aligned = reinterpret_cast<uintptr_t>(d0) % 4 == 0;  // K + 4 is a multiple of 4
  for (int s = 0; s < 3; ++s) {
    uint8_t* d = d0 + s * (K + 4);
    for (int i = tid; i < K / 4; i += kEncThreads) {
      const uint32_t v = spread4(out[s][i >> 3] >> (4 * (i & 7)));
      if (aligned) {
        reinterpret_cast<uint32_t*>(d)[i] = v;
      } else {
        for (int k = 0; k < 4; ++k) d[4 * i + k] = static_cast<uint8_t>(v >> (8 * k));
      }
    }
  }
  if (tid != 0) return;
  // the tail multiplexing of lte_turbo.cpp:664-677
  uint8_t ts[2][3], tp[2][3];
  for (int e = 0; e < 2; ++e) {
    const auto fb = [&](int i) { return f[e][(i >> 5) + 1] >> (i & 31) & 1u; };
    uint8_t s = static_cast<uint8_t>(fb(K - 1) << 2 | fb(K - 2) << 1 | fb(K - 3));
    for (int i = 0; i < 3; ++i) {
      ts[e][i] = ((s >> 1) & 1u) ^ ((s >> 2) & 1u);  // the input that zeroes the feedback
      tp[e][i] = rsc_step(s, ts[e][i]);
    }
  }
  d0[K] = ts[0][0]; d0[K + 1] = tp[0][1]; d0[K + 2] = ts[0][1]; d0[K + 3] = tp[0][2];
  d1[K] = tp[0][0]; d1[K + 1] = ts[0][1]; d1[K + 2] = tp[0][2]; d1[K + 3] = ts[1][0];
  d2[K] = tp[1][0]; d2[K + 1] = ts[1][1]; d2[K + 2] = tp[1][1]; d2[K + 3] = ts[1][2];
}

// BPSK over AWGN: one Box-Muller draw per encoded bit from two counter-derived uniforms (the
// host's awgn_llr), LLR = 2 y / sigma^2; filler positions of d0 and d1 get 0.
__global__ void __launch_bounds__(kGenThreads) awgn_kernel(const GenBlock* __restrict__ blocks,
                                                          const uint8_t* __restrict__ d012,
                                                          float* __restrict__ llr) {
  const GenBlock b = blocks[blockIdx.x];
  const uint64_t key = mix64((b.seed ^ 0x2545f4914f6cdd1dull) ^ 0xbb67ae8584caa73bull);
  const int n = 3 * (b.k + 4);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const uint64_t c = static_cast<uint64_t>(i);
    // every product and sum rounded on its own (no contraction into FMA), as on the host
    const double u1 = __dmul_rn(__dadd_rn(static_cast<double>(mix64(key + 2 * c) >> 11), 0.5), 0x1.0p-53);
    const double u2 = __dmul_rn(__dadd_rn(static_cast<double>(mix64(key + 2 * c + 1) >> 11), 0.5), 0x1.0p-53);
    const double z = __dmul_rn(sqrt(__dmul_rn(-2.0, log(u1))), cos(__dmul_rn(6.283185307179586, u2)));
    const double y = __dadd_rn(d012[b.llr + i] ? 1.0 : -1.0, __dmul_rn(b.sigma, z));
    const int lane_pos = i % (b.k + 4);
    const bool filler = i < 2 * (b.k + 4) && lane_pos < b.filler;
    llr[b.llr + i] = filler ? 0.0f : __double2float_rn(__dmul_rn(b.scale, y));
  }
}

constexpr int kRmGenThreads = 512;

struct RmGen {
  int32_t k, filler, e, rv;
  int64_t e_off, d_off;
};

// One CTA per block: output bit kk is the stream bit at the kk-th <NULL>-free position of the
// circular walk from k0 (wrapping), i.e. the valid position of rank (rank(k0) + kk) mod Nv.  The
// encoded bits go to shared memory by rank (closed form), the output is read from there in order:
// every global access walks its array.  Bound by the index arithmetic of the rank; 4096 mixed blocks at
// rate 1/2: 134 us, 170 us with a scan over the positions and a scattered byte store per bit.
__global__ void __launch_bounds__(kRmGenThreads) rate_match_kernel(const RmGen* __restrict__ blocks,
                                                                  const uint8_t* __restrict__ d012,
                                                                  uint8_t* __restrict__ e_bits) {
  __shared__ int tables[kRankTableInts];
  __shared__ uint8_t by_rank[3 * (6144 + 4)];
  const RmGen b = blocks[blockIdx.x];
  CircularRank cr(b.k, b.filler, tables);
  cr.setup();
  __syncthreads();
  const uint8_t* src = d012 + b.d_off;
  const int n = 3 * cr.d;
  for (int i = threadIdx.x; i < n; i += kRmGenThreads) {
    const int r = cr.rank_of_element(i);
    if (r >= 0) by_rank[r] = src[i];
  }
  __syncthreads();
  const int nv = cr.valid(), r0 = cr.rank(cr.k0(b.rv));
  uint8_t* out = e_bits + b.e_off;
  // 4 output bits per thread and step, from the first 4-byte boundary on
  const int head = min(b.e, static_cast<int>(-reinterpret_cast<intptr_t>(out) & 3));
  const int quads = (b.e - head) / 4;
  int at = (r0 + head + 4 * static_cast<int>(threadIdx.x)) % nv;
  const int step = 4 * kRmGenThreads % nv;
  for (int i = threadIdx.x; i < quads; i += kRmGenThreads) {
    uint32_t v = 0;
    int a = at;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v |= static_cast<uint32_t>(by_rank[a]) << (8 * k);
      if (++a == nv) a = 0;
    }
    *reinterpret_cast<uint32_t*>(out + head + 4 * i) = v;
    at += step;
    if (at >= nv) at -= nv;
  }
  const int rest = head + 4 * quads;  // what is left: the head and up to 3 bits behind the quads
  const int left = head + b.e - rest;
  if (static_cast<int>(threadIdx.x) < left) {
    const int kk = static_cast<int>(threadIdx.x) < head ? threadIdx.x : rest + threadIdx.x - head;
    out[kk] = by_rank[(r0 + kk) % nv];
  }
}

template <class T>
T* reserve(DeviceBuffer& b, size_t count) {
  b.reserve(count * sizeof(T));
  return static_cast<T*>(b.ptr);
}

}  // namespace

void Decoder::awgn_code_blocks_device(uint64_t seed, size_t n, const int32_t* k,
                                      const int32_t* filler, const float* ebn0_db, bool crc24b,
                                      uint8_t* bits, float* llr, void* stream) {
  std::lock_guard<std::mutex> lock(mu_);
  ok(cudaSetDevice(device_), "cudaSetDevice");
  if (n == 0) return;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  std::vector<GenBlock> v(n);
  std::vector<int32_t> tab(n);
  int64_t boff = 0, loff = 0;
  for (size_t i = 0; i < n; ++i) {
    if (qpp_index(k[i]) < 0) throw OutOfRange("unsupported QPP block size");
    if (filler[i] < 0 || filler[i] >= k[i] || (crc24b && filler[i] + 24 >= k[i]))
      throw InvalidArgument("invalid filler count");
    GenBlock& g = v[i];
    g.k = k[i];
    g.filler = filler[i];
    g.bits = boff;
    g.llr = loff;
    g.seed = host_mix64(seed + 0x51ed270b27ull * (i + 1));
    // the host generator's channel parameters, computed the same way
    const double rate = static_cast<double>(k[i]) / (3.0 * (k[i] + 4));
    const double sigma2 = 1.0 / (2.0 * rate * std::pow(10.0, ebn0_db[i] / 10.0));
    g.sigma = std::sqrt(sigma2);
    g.scale = 2.0 / sigma2;
    tab[i] = table_offset(k[i]);
    boff += k[i];
    loff += 3 * static_cast<int64_t>(k[i] + 4);
  }
  order_after_previous(stream);
  GenBlock* dv = reserve<GenBlock>(d_gen_, n);
  int32_t* dt = reserve<int32_t>(d_gentab_, n);
  uint8_t* enc = reserve<uint8_t>(d_genenc_, static_cast<size_t>(loff));
  upload(dv, v.data(), n * sizeof(GenBlock), stream);
  upload(dt, tab.data(), n * sizeof(int32_t), stream);
  gen_bits_kernel<<<static_cast<unsigned>(n), kGenThreads, 0, st>>>(
      dv, crc24b ? 1 : 0, static_cast<const uint32_t*>(d_xpow_.ptr), bits);
  ok(cudaGetLastError(), "bit generation launch");
  encode_kernel<<<static_cast<unsigned>(n), kEncThreads, 0, st>>>(
      dv, perm_table(), dt, bits, enc);
  ok(cudaGetLastError(), "encoder launch");
  awgn_kernel<<<static_cast<unsigned>(n), kGenThreads, 0, st>>>(dv, enc, llr);
  ok(cudaGetLastError(), "channel launch");
  timing_.launches += 3;
  mark_done(stream);
}

void Decoder::turbo_encode_device(size_t n, const int32_t* k, const int32_t* filler,
                                  const uint8_t* bits, uint8_t* d012, void* stream) {
  std::lock_guard<std::mutex> lock(mu_);
  ok(cudaSetDevice(device_), "cudaSetDevice");
  if (n == 0) return;
  std::vector<GenBlock> v(n);
  std::vector<int32_t> tab(n);
  int64_t boff = 0, loff = 0;
  for (size_t i = 0; i < n; ++i) {
    if (qpp_index(k[i]) < 0) throw OutOfRange("unsupported QPP block size");
    if (filler[i] < 0 || filler[i] >= k[i]) throw InvalidArgument("invalid filler count");
    v[i] = GenBlock{k[i], filler[i], boff, loff, 0, 0.0, 0.0};
    tab[i] = table_offset(k[i]);
    boff += k[i];
    loff += 3 * static_cast<int64_t>(k[i] + 4);
  }
  order_after_previous(stream);
  GenBlock* dv = reserve<GenBlock>(d_gen_, n);
  int32_t* dt = reserve<int32_t>(d_gentab_, n);
  upload(dv, v.data(), n * sizeof(GenBlock), stream);
  upload(dt, tab.data(), n * sizeof(int32_t), stream);
  encode_kernel<<<static_cast<unsigned>(n), kEncThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      dv, perm_table(), dt, bits, d012);
  ok(cudaGetLastError(), "encoder launch");
  timing_.launches += 1;
  mark_done(stream);
}

void Decoder::rate_match_device(size_t n, const RmBlockDesc* blocks, const uint8_t* d012,
                                size_t d012_len, uint8_t* e_bits, size_t e_len, void* stream) {
  std::lock_guard<std::mutex> lock(mu_);
  ok(cudaSetDevice(device_), "cudaSetDevice");
  if (n == 0) return;
  std::vector<RmGen> v(n);
  for (size_t i = 0; i < n; ++i) {
    const RmBlockDesc& b = blocks[i];
    if (qpp_index(b.k) < 0) throw OutOfRange("unsupported QPP block size");
    if (b.filler < 0 || b.filler >= b.k || b.rv > 3 || b.e < 0)
      throw InvalidArgument("invalid filler count, rv or E");
    if (b.e_offset < 0 || static_cast<size_t>(b.e_offset) + static_cast<size_t>(b.e) > e_len)
      throw InvalidArgument("rate-matched bits out of range");
    if (b.llr_offset < 0 ||
        static_cast<size_t>(b.llr_offset) + 3 * static_cast<size_t>(b.k + 4) > d012_len)
      throw InvalidArgument("encoded bits out of range");
    v[i] = RmGen{b.k, b.filler, b.e, static_cast<int32_t>(b.rv), b.e_offset, b.llr_offset};
  }
  order_after_previous(stream);
  RmGen* dv = reserve<RmGen>(d_genrm_, n);
  upload(dv, v.data(), n * sizeof(RmGen), stream);
  rate_match_kernel<<<static_cast<unsigned>(n), kRmGenThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      dv, d012, e_bits);
  ok(cudaGetLastError(), "rate matching launch");
  timing_.launches += 1;
  mark_done(stream);
}

}  // namespace tcb
