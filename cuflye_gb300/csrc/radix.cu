// radix.cu — stable least-significant-digit radix sort of (u64 key, u64 value)
// pairs, 8 bits per pass, over a chosen list of digits (value bytes 0-7 are
// digits 0-7, key bytes are digits 8-15).  Builds the k-mer index.
//
// A pass counts each tile's digits, scans the counts (digit-major) over the
// whole device and scatters.  The scatter stages its tile in shared memory in
// digit order, so that each digit's pairs leave as one run (4,096 pairs a tile:
// 16 pairs, 256 bytes, a digit on average) and two blocks of 512 threads
// share an SM.  40e6 pairs: 0.41 ms a pass, 40 bytes a pair at 3.9 TB/s (a
// single-block scan and unstaged stores before: 3.1 ms).
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "kernels.h"

namespace cuflye {
namespace {

constexpr int kRadixBlock = 512;
constexpr int kRadixWarps = kRadixBlock / 32;
constexpr int kRadixItems = 8;  // pairs per thread
constexpr uint32_t kRadixTile = kRadixBlock * kRadixItems;
constexpr uint32_t kRadixWarpTile = 32 * kRadixItems;  // consecutive pairs of a warp

__device__ __forceinline__ uint32_t digit_of(uint64_t key, uint64_t val, int d) {
  // digits 0..7: value bytes (least significant first); 8..15: key bytes
  return d < 8 ? static_cast<uint32_t>((val >> (8 * d)) & 0xffu)
               : static_cast<uint32_t>((key >> (8 * (d - 8))) & 0xffu);
}

__global__ void __launch_bounds__(kRadixBlock) radix_histogram(
    const uint64_t* __restrict__ words, uint64_t n, int shift, uint32_t* __restrict__ hist,
    uint32_t ntiles) {
  __shared__ uint32_t h[256];
  if (threadIdx.x < 256) h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t t0 = static_cast<uint64_t>(blockIdx.x) * kRadixTile;
  uint32_t d[kRadixItems];
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    const uint64_t i = t0 + r * kRadixBlock + threadIdx.x;
    d[r] = i < n ? static_cast<uint32_t>(words[i] >> shift) & 0xffu : 256u;
  }
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r)
    if (d[r] < 256u) atomicAdd(&h[d[r]], 1u);
  __syncthreads();
  if (threadIdx.x < 256)
    hist[static_cast<uint64_t>(threadIdx.x) * ntiles + blockIdx.x] = h[threadIdx.x];
}

struct RadixSmem {
  uint64_t key[kRadixTile];  // the tile's pairs in digit order
  uint64_t val[kRadixTile];
  uint64_t gbase[256];               // each digit's first output slot of the tile
  uint32_t wc[kRadixWarps][256];     // per-warp digit counts, then offsets
  uint32_t dbase[256];               // tile-local start of each digit
  uint32_t ws[8];
};

// Stable: warp w owns the tile's pairs [w * 256, (w + 1) * 256), visited in
// rounds of 32; match_any ranks a round, per-warp counters carry the ranks
// across rounds, and a scan over warps places each digit's pairs in order.
__global__ void __launch_bounds__(kRadixBlock, 2) radix_scatter(
    const uint64_t* __restrict__ keys_in, const uint64_t* __restrict__ vals_in,
    uint64_t* __restrict__ keys_out, uint64_t* __restrict__ vals_out, uint64_t n, int d,
    const uint64_t* __restrict__ offs, uint32_t ntiles) {
  extern __shared__ __align__(16) unsigned char radix_raw[];
  RadixSmem& sm = *reinterpret_cast<RadixSmem*>(radix_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint64_t t0 = static_cast<uint64_t>(blockIdx.x) * kRadixTile;
  const uint32_t tn = static_cast<uint32_t>(min(static_cast<uint64_t>(kRadixTile), n - t0));
  for (int i = threadIdx.x; i < kRadixWarps * 256; i += kRadixBlock) (&sm.wc[0][0])[i] = 0;
  if (threadIdx.x < 256)
    sm.gbase[threadIdx.x] = offs[static_cast<uint64_t>(threadIdx.x) * ntiles + blockIdx.x];
  uint64_t k[kRadixItems], v[kRadixItems];
  uint32_t rk[kRadixItems];
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    const uint32_t j = warp * kRadixWarpTile + r * 32 + lane;
    k[r] = j < tn ? keys_in[t0 + j] : 0;
    v[r] = j < tn ? vals_in[t0 + j] : 0;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    const uint32_t j = warp * kRadixWarpTile + r * 32 + lane;
    const bool valid = j < tn;
    const uint32_t dig = valid ? digit_of(k[r], v[r], d) : 256u;
    const uint32_t peers = __match_any_sync(0xffffffffu, dig);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (valid && lane == leader) {
      base = sm.wc[warp][dig];
      sm.wc[warp][dig] = base + __popc(peers);
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    rk[r] = base + __popc(peers & lt);
    __syncwarp();
  }
  __syncthreads();
  uint32_t tot = 0, inc = 0;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int w = 0; w < kRadixWarps; ++w) {
      const uint32_t c = sm.wc[w][threadIdx.x];
      sm.wc[w][threadIdx.x] = tot;
      tot += c;
    }
    inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) sm.ws[warp] = inc;
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += sm.ws[w];
    sm.dbase[threadIdx.x] = before + inc - tot;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    const uint32_t j = warp * kRadixWarpTile + r * 32 + lane;
    if (j < tn) {
      const uint32_t dig = digit_of(k[r], v[r], d);
      const uint32_t p = sm.dbase[dig] + sm.wc[warp][dig] + rk[r];
      sm.key[p] = k[r];
      sm.val[p] = v[r];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    const uint32_t j = r * kRadixBlock + threadIdx.x;
    if (j < tn) {
      const uint64_t kk = sm.key[j], vv = sm.val[j];
      const uint32_t dig = digit_of(kk, vv, d);
      const uint64_t dst = sm.gbase[dig] + (j - sm.dbase[dig]);
      keys_out[dst] = kk;
      vals_out[dst] = vv;
    }
  }
}

uint64_t radix_tiles(uint64_t n) { return (n + kRadixTile - 1) / kRadixTile; }

}  // namespace

// The scratch: 256 counts a tile, their offsets (8 bytes each), the scan's.
size_t radix_hist_words(uint64_t n) {
  const uint64_t c = 256 * radix_tiles(n);
  return 3 * c + 2 * scan_temp_words(c) + 4;
}

cudaError_t radix_sort_pairs(uint64_t* keys, uint64_t* vals, uint64_t* keys_alt,
                             uint64_t* vals_alt, uint64_t n, const int* digits, int ndigits,
                             uint32_t* hist, int* result_in_alt, cudaStream_t stream) {
  const uint64_t nt = radix_tiles(n);
  if (nt >= (1ull << 31)) return cudaErrorInvalidValue;
  const uint32_t ntiles = static_cast<uint32_t>(nt);
  const uint64_t c = 256 * nt;  // even: the offsets are 8-byte aligned
  uint64_t* offs = reinterpret_cast<uint64_t*>(hist + c);
  uint64_t* temp = offs + c + 1;
  cudaError_t e = cudaFuncSetAttribute(radix_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(sizeof(RadixSmem)));
  if (e != cudaSuccess) return e;
  uint64_t *ki = keys, *vi = vals, *ko = keys_alt, *vo = vals_alt;
  for (int p = 0; p < ndigits; ++p) {
    const int d = digits[p];
    count_launch();
    radix_histogram<<<ntiles, kRadixBlock, 0, stream>>>(d < 8 ? vi : ki, n, 8 * (d & 7), hist,
                                                        ntiles);
    e = exclusive_scan_u32_to_u64(hist, offs, c, temp, stream);
    if (e != cudaSuccess) return e;
    count_launch();
    radix_scatter<<<ntiles, kRadixBlock, sizeof(RadixSmem), stream>>>(ki, vi, ko, vo, n, d, offs,
                                                                      ntiles);
    std::swap(ki, ko);
    std::swap(vi, vo);
  }
  *result_in_alt = (ki == keys_alt);
  return cudaGetLastError();
}

}  // namespace cuflye
