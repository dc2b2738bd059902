// util.cu — exclusive prefix sums and 2-bit packing.
#include <atomic>
#include <cstdint>

#include "common.cuh"
#include "kernels.h"

namespace cuflye {

static std::atomic<unsigned long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
unsigned long long launches_total() { return g_launches.load(std::memory_order_relaxed); }

namespace {

constexpr int kScanBlock = 256;
constexpr int kScanItems = 8;
constexpr uint64_t kScanTile = kScanBlock * kScanItems;

template <typename In>
__global__ void scan_tile_sums(const In* __restrict__ in, uint64_t n, uint64_t* __restrict__ sums) {
  __shared__ uint64_t ws[kScanBlock / 32];
  const uint64_t t0 = static_cast<uint64_t>(blockIdx.x) * kScanTile;
  uint64_t s = 0;
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = t0 + static_cast<uint64_t>(j) * kScanBlock + threadIdx.x;
    if (i < n) s += static_cast<uint64_t>(in[i]);
  }
  for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t t = 0;
    for (int w = 0; w < kScanBlock / 32; ++w) t += ws[w];
    sums[blockIdx.x] = t;
  }
}

// Single-block exclusive scan of the tile sums (sums[ntiles] = grand total).
__global__ void scan_sums(uint64_t* sums, uint64_t ntiles) {
  __shared__ uint64_t ws[32];
  __shared__ uint64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = blockDim.x / 32;
  for (uint64_t base = 0; base < ntiles; base += blockDim.x) {
    const uint64_t i = base + threadIdx.x;
    const uint64_t v = i < ntiles ? sums[i] : 0;
    uint64_t inc = v;
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t o = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += o;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const uint64_t w = lane < nw ? ws[lane] : 0;
      uint64_t wi = w;
      for (int d = 1; d < 32; d <<= 1) {
        const uint64_t o = __shfl_up_sync(0xffffffffu, wi, d);
        if (lane >= d) wi += o;
      }
      if (lane < nw) ws[lane] = wi - w;
    }
    __syncthreads();
    const uint64_t ex = carry + ws[warp] + inc - v;
    if (i < ntiles) sums[i] = ex;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = ex + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[ntiles] = carry;
}

// Short arrays: one block a scan (the second's for a pair of them), so that a
// small call pays one launch, not three.
constexpr int kSmallBlock = 1024;
constexpr uint64_t kSmallScan = 32768;

__global__ void __launch_bounds__(kSmallBlock) scan_small(const uint32_t* __restrict__ in0,
                                                          uint64_t* __restrict__ out0,
                                                          const uint32_t* __restrict__ in1,
                                                          uint64_t* __restrict__ out1,
                                                          uint32_t n) {
  __shared__ uint64_t ws[kSmallBlock / 32];
  const uint32_t* __restrict__ in = blockIdx.x ? in1 : in0;
  uint64_t* __restrict__ out = blockIdx.x ? out1 : out0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t carry = 0;
  for (uint32_t t0 = 0; t0 < n; t0 += kSmallBlock * 4) {
    const uint32_t a = t0 + threadIdx.x * 4;
    uint32_t v[4];
    uint64_t s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[j] = a + j < n ? in[a + j] : 0u;
      s += v[j];
    }
    uint64_t inc = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t o = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += o;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    uint64_t before = carry, all = 0;
#pragma unroll
    for (int w = 0; w < kSmallBlock / 32; ++w) {
      const uint64_t x = ws[w];
      before += w < warp ? x : 0;
      all += x;
    }
    uint64_t run = before + inc - s;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (a + j < n) out[a + j] = run;
      run += v[j];
    }
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
}

template <typename In>
__global__ void scan_downsweep(const In* __restrict__ in, uint64_t* __restrict__ out, uint64_t n,
                               const uint64_t* __restrict__ sums) {
  __shared__ uint64_t ws[kScanBlock / 32 + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t t0 = static_cast<uint64_t>(blockIdx.x) * kScanTile;
  // each thread owns kScanItems consecutive elements
  const uint64_t a = t0 + static_cast<uint64_t>(threadIdx.x) * kScanItems;
  uint64_t v[kScanItems];
  uint64_t s = 0;
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = a + j;
    v[j] = i < n ? static_cast<uint64_t>(in[i]) : 0;
    s += v[j];
  }
  uint64_t inc = s;
  for (int d = 1; d < 32; d <<= 1) {
    const uint64_t o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t c = 0;
    for (int w = 0; w < kScanBlock / 32; ++w) {
      const uint64_t t = ws[w];
      ws[w] = c;
      c += t;
    }
  }
  __syncthreads();
  uint64_t run = sums[blockIdx.x] + ws[warp] + inc - s;
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = a + j;
    if (i < n) out[i] = run;
    run += v[j];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = sums[gridDim.x];
}

// The codes of four letters (ACGT, either case), the first most significant;
// other: nonzero afterwards when any character is something else.  Bits 1-2 of
// a letter tell it (A 0, C 1, T 2, G 3); the letter that they stand for is looked
// up and compared.  15 instructions for four bases, where a switch takes 8 a base.
__device__ __forceinline__ uint32_t pack4(uint32_t w, uint32_t& other) {
  const uint32_t t = (w >> 1) & 0x03030303u;
  const uint32_t code = t ^ ((t >> 1) & 0x01010101u);
  const uint32_t nibbles = __byte_perm(code | code >> 4, 0, 0x0020) & 0xffffu;
  other |= (w & 0xdfdfdfdfu) ^ __byte_perm(0x54474341u, 0, nibbles);
  return code * 0x40100401u >> 24;  // two-bit fields that do not meet below bit 24
}

__global__ void pack_kernel(const uint8_t* __restrict__ ascii, uint64_t nbases,
                            uint64_t* __restrict__ words, uint64_t nwords) {
  const uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= nwords) return;
  const uint64_t b0 = w * 32;
  uint64_t x = 0;
  if (b0 + 32 <= nbases) {
    const uint4* p = reinterpret_cast<const uint4*>(ascii + b0);
    uint4 c[2];
    if ((reinterpret_cast<uintptr_t>(ascii + b0) & 15u) == 0) {
      c[0] = p[0];
      c[1] = p[1];
    } else {
      uint8_t* cb = reinterpret_cast<uint8_t*>(c);
      for (int i = 0; i < 32; ++i) cb[i] = ascii[b0 + i];
    }
    const uint32_t* cw = reinterpret_cast<const uint32_t*>(c);
    uint32_t other = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) x = x << 8 | pack4(cw[i], other);
    if (other) {  // characters besides the four letters: code 0
      const uint8_t* cb = reinterpret_cast<const uint8_t*>(c);
      x = 0;
      for (int i = 0; i < 32; ++i) x = (x << 2) | base_code(cb[i]);
    }
  } else {
    for (int i = 0; i < 32; ++i) {
      const uint64_t b = b0 + i;
      x = (x << 2) | (b < nbases ? base_code(ascii[b]) : 0u);
    }
  }
  words[w] = x;
}

}  // namespace

size_t scan_temp_words(uint64_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

cudaError_t exclusive_scan_u32_to_u64(const uint32_t* in, uint64_t* out, uint64_t n,
                                      uint64_t* temp, cudaStream_t s) {
  if (n == 0) return cudaMemsetAsync(out, 0, sizeof(uint64_t), s);
  if (n <= kSmallScan) {
    count_launch();
    scan_small<<<1, kSmallBlock, 0, s>>>(in, out, in, out, static_cast<uint32_t>(n));
    return cudaGetLastError();
  }
  const uint64_t ntiles = (n + kScanTile - 1) / kScanTile;
  count_launch();
  scan_tile_sums<uint32_t><<<static_cast<unsigned>(ntiles), kScanBlock, 0, s>>>(in, n, temp);
  count_launch();
  scan_sums<<<1, 1024, 0, s>>>(temp, ntiles);
  count_launch();
  scan_downsweep<uint32_t><<<static_cast<unsigned>(ntiles), kScanBlock, 0, s>>>(in, out, n, temp);
  return cudaGetLastError();
}

cudaError_t exclusive_scan_pair(const uint32_t* in0, uint64_t* out0, const uint32_t* in1,
                                uint64_t* out1, uint64_t n, uint64_t* temp, cudaStream_t s) {
  if (n == 0 || n > kSmallScan) {
    const cudaError_t e = exclusive_scan_u32_to_u64(in0, out0, n, temp, s);
    return e != cudaSuccess ? e : exclusive_scan_u32_to_u64(in1, out1, n, temp, s);
  }
  count_launch();
  scan_small<<<2, kSmallBlock, 0, s>>>(in0, out0, in1, out1, static_cast<uint32_t>(n));
  return cudaGetLastError();
}

cudaError_t pack_bases(const uint8_t* ascii, uint64_t nbases, uint64_t* words, cudaStream_t s) {
  const uint64_t nwords = (nbases + 31) / 32 + 1;
  count_launch();
  pack_kernel<<<static_cast<unsigned>((nwords + 255) / 256), 256, 0, s>>>(ascii, nbases, words,
                                                                         nwords);
  return cudaGetLastError();
}

}  // namespace cuflye
