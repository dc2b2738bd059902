// runs.cu — candidate hits found, sorted and filtered as runs.
//
// Hits of one (query, target) pair come in runs at consecutive cur and ext
// positions: a window's hit (id, pos) continues the run of the window before
// it exactly when that window is solid and the base before the k-mer is the
// same in query and target.  So the index keeps, for every stored entry, the
// bases around its k-mer (one byte), and a query window finds the runs that
// start in its bucket by comparing bytes; a hit inside a run costs that byte
// and is never written.  A run's length is how far the packed query and target
// agree, cut at the query's next window that is not solid.
//
// The runs are sorted like hits (radix sort by ext id of runs generated in
// window order), grouped by ext id, and each group's prefilter is decided from
// its runs.  run_chain.cu chains them.
//
// Measured on all reads of a 5 Mb genome at 40x (HiFi, k = 17: 7.2e9 hits in
// 36e6 runs, 64 GiB budget): hit generation 183 -> 4.9 ms, KmerMatch sort 54 ->
// 2.0 ms, groups 51 -> 3.9 ms, DP 50 -> 2.1 ms, backtrack 27 -> 3.3 ms against
// writing, sorting and chaining every hit (the hit path, which remains for what
// the run path leaves open and for indexes without its tables).  At 6 % error (3
// Mb genome, 30x ONT reads: 4.7e8 hits in 59e6 runs) 50 -> 8.6 ms without open
// groups, 11 to 20 with them.  One read: 1.0 -> 0.24 ms, its groups' serial scans
// being as many times shorter as its runs are long.
//
// Needs an odd k: an even k has k-mers equal to their own reverse complement,
// stored on one strand only, so that a run on the other strand has holes.  Short
// k-mers (below kRunLeastK in api.cu) stay with the hit path, which is faster there.
#include <algorithm>
#include <climits>
#include <cstdint>

#include "common.cuh"
#include "hits.cuh"
#include "kernels.h"
#include "proposals.cuh"
#include "runs.h"

namespace cuflye {
namespace {

inline unsigned grid(uint64_t n, int b) {
  return static_cast<unsigned>((n + b - 1) / b > 0 ? (n + b - 1) / b : 1);
}

constexpr uint8_t kWinSolid = 8;  // window flag beside kWinRev and kWinFiltered

__device__ __forceinline__ uint32_t base_at(const uint64_t* __restrict__ words, uint64_t g) {
  return static_cast<uint32_t>(__ldg(words + (g >> 5)) >> (62 - 2 * (g & 31))) & 3u;
}

// 32 bases from base g on (g >= 0; two words).
__device__ __forceinline__ uint64_t bases32(const uint64_t* __restrict__ words, uint64_t g) {
  const uint64_t hi = __ldg(words + (g >> 5));
  const uint32_t s = static_cast<uint32_t>(g & 31u);
  return s ? (hi << (2 * s)) | (__ldg(words + (g >> 5) + 1) >> (64 - 2 * s)) : hi;
}

__global__ void neighbour_kernel(const uint64_t* __restrict__ pos, uint64_t n,
                                 const uint64_t* __restrict__ words,
                                 const uint64_t* __restrict__ base_off,
                                 const int32_t* __restrict__ slot_len, int k,
                                 uint8_t* __restrict__ nbr) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t v = pos[i];
  const uint32_t sid = static_cast<uint32_t>(v >> 32);
  const int32_t sp = static_cast<int32_t>(v & 0xffffffffu);
  const int32_t len = slot_len[sid >> 1];
  const uint64_t b = base_off[sid >> 1];
  const int32_t p = (sid & 1u) ? len - sp - k : sp;  // the window on the forward strand
  uint32_t before = 4, after = 4;
  if (p > 0) before = base_at(words, b + static_cast<uint64_t>(p) - 1);
  if (p + k < len) after = base_at(words, b + static_cast<uint64_t>(p) + k);
  if (sid & 1u) {
    const uint32_t x = before;
    before = after == 4 ? 4u : 3u - after;
    after = x == 4 ? 4u : 3u - x;
  }
  nbr[i] = static_cast<uint8_t>(before | (after << 4));
}

// What a bucket entry's neighbour nibble must be for its hit to continue the
// run of the window before (7 matches no entry), and where the nibble sits in
// the entry's byte: the base before the window, on the entry's strand (the
// complement of it after the k-mer when the lookup flips).
struct RunTest {
  uint32_t expect;
  int shift;  // 0, or 4 when the lookup flips
};

// What the emission reads of a window that starts runs or is filtered:
// {table word (8 bytes), the window's position in its query, own entry | expect
// << 22 | flip << 25}.  Own entry: its place in the bucket, kNoSelf without one.
constexpr uint32_t kNoSelf = (1u << kCountBits) - 1;
static_assert(kCountBits == 22, "bucket places take 22 bits of a window record");

__device__ __forceinline__ uint32_t bucket_size(uint64_t meta) {
  return static_cast<uint32_t>((meta >> 40) & ((1ULL << kCountBits) - 1));
}

// Which of 16 entries' nibbles differ from the pattern: bit 8 j + 7 - s for
// entry 4 s + j (byte j of word s), so that one popcount counts them all.
__device__ __forceinline__ uint32_t differ16(uint4 x, int shift, uint32_t pat) {
  auto word = [&](uint32_t w) {
    return ((((w >> shift) & 0x0f0f0f0fu) ^ pat) + 0x7f7f7f7fu) & 0x80808080u;
  };
  return word(x.x) | (word(x.y) >> 1) | (word(x.z) >> 2) | (word(x.w) >> 3);
}
// The entries from lo on (0..16) in that order of bits.
__device__ __forceinline__ uint32_t entries_from(uint32_t lo) {
  const uint32_t s = lo >> 2, top = 0x80u >> s;
  return lo >= 16 ? 0u
                  : ((top - 1u) & 0xf0u) * 0x01010101u |
                        ((top * 0x01010101u) & (0xffffffffu << (8 * (lo & 3u))));
}

// Entries of the bucket [off, off + c) that start a run (the query's own
// entry among them): 16 entries a load, four loads issued together.
__device__ __forceinline__ uint32_t count_starts(const DeviceIndex& idx, uint64_t off, uint32_t c,
                                                 RunTest rt) {
  const uint32_t pat = rt.expect * 0x01010101u;
  const uint4* nb = reinterpret_cast<const uint4*>(idx.nbr);
  const uint64_t c0 = off >> 4, c1 = (off + c - 1) >> 4;
  const uint32_t head = entries_from(static_cast<uint32_t>(off & 15)),
                 tail = ~entries_from(static_cast<uint32_t>((off + c - 1) & 15) + 1);
  uint32_t ns = 0;
  for (uint64_t b = c0; b <= c1; b += 4) {
    uint4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (b + u <= c1) x[u] = __ldg(nb + b + u);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (b + u <= c1) {
        uint32_t m = differ16(x[u], rt.shift, pat);
        if (b + u == c0) m &= head;
        if (b + u == c1) m &= tail;
        ns += __popc(m);
      }
    }
  }
  return ns;
}

// What most entries of a window's bucket have on the side that tells whether
// they continue a run (a nibble's value, 7: not known), and how many differ.
struct BucketSide {
  uint32_t most, others;
};

__device__ __forceinline__ BucketSide record_side(const uint4& rec, bool rev) {
  return BucketSide{rec.z >> (kCountBits + (rev ? 3 : 0)) & 7u, rec.w >> (rev ? 16 : 0) & 0xfffu};
}

// A window's table word, its own entry's place in the bucket, the bucket's side
// and the flags.
__device__ __forceinline__ uint8_t probe_run_window(const DeviceIndex& idx, const QueryBatch& q,
                                                    uint32_t qi, uint64_t p, uint64_t& meta,
                                                    uint32_t& self, BucketSide& side) {
  const WindowKmer km = window_kmer(q, qi, p, idx.k);
  const int32_t qdi = q.qdi[qi];
  uint4 rec;
  const bool own = own_window(idx, qdi, p, km.x, rec), recorded = own && idx.windows;
  bool found = rec.w & kWindowFound;
  meta = recorded ? static_cast<uint64_t>(rec.y) << 32 | rec.x
                  : index_probe(idx, km.key, &found);
  uint8_t fl = km.rev ? kWinRev : 0;
  self = kNoSelf;
  side = BucketSide{7, 0};
  if (!found) return fl;
  if (meta & kRepetitiveBit) return fl | kWinFiltered;
  fl |= kWinSolid;
  if (recorded) {
    self = rec.z & kPlaceMask;
    side = record_side(rec, km.rev);
  } else if (own) {
    self = bucket_find(idx, meta & kOffsetMask, bucket_size(meta),
                       self_entry(idx, qdi, p, km.rev));
  }
  return fl;
}

// The base before the query's own window p in its target (4: the target's end):
// what its entry's nibble says, in step with the query's bases.
__device__ __forceinline__ uint32_t own_before(const DeviceIndex& idx, int32_t qdi, uint64_t p) {
  const uint32_t slot = static_cast<uint32_t>(qdi) >> 1;
  const int64_t f = forward_window(idx, qdi, p);
  const uint64_t b = idx.tbase[slot];
  if (!(qdi & 1)) return f > 0 ? base_at(idx.twords, b + static_cast<uint64_t>(f) - 1) : 4u;
  const int64_t after = f + idx.k;
  return after < idx.slot_len[slot]
             ? 3u - base_at(idx.twords, b + static_cast<uint64_t>(after)) : 4u;
}

// Bases x .. x + 31 of a target strand (first base tbase, tlen bases).
__device__ __forceinline__ uint64_t target_bases32(const uint64_t* __restrict__ words,
                                                   uint64_t tbase, int32_t tlen, bool rev,
                                                   int32_t x) {
  if (!rev) return bases32(words, tbase + static_cast<uint64_t>(x));
  // the reverse complement of the 32 forward bases that end before len - x
  const int64_t s = static_cast<int64_t>(tbase) + tlen - 32 - x;
  const uint64_t f = s >= 0 ? bases32(words, static_cast<uint64_t>(s))
                            : bases32(words, 0) >> (2 * -s);
  return revcomp(f, 32);
}

// Whether windows [w0, w1) of query qi (and the one before) are those of the
// indexed target of its id, base for base (called by the whole block).  Their
// records then tell all that a probe would, strand and neighbours included.
__device__ __forceinline__ bool indexed_windows(const DeviceIndex& idx, const QueryBatch& q,
                                                uint32_t qi, uint64_t w0, uint64_t w1) {
  const int32_t qdi = q.qdi[qi];
  bool differ = true;
  if (idx.windows && idx.twords && qdi >= 0) {
    const uint32_t slot = static_cast<uint32_t>(qdi) >> 1;
    const int32_t len = idx.slot_len[slot];
    const int64_t p0 = static_cast<int64_t>(w0 - q.win_off[qi]);
    const int64_t b0 = p0 > 0 ? p0 - 1 : 0, b1 = static_cast<int64_t>(w1 - q.win_off[qi]) + idx.k - 1;
    differ = b1 > len;
    for (int64_t x = b0 + 32 * threadIdx.x; !differ && x < b1; x += 32 * blockDim.x) {
      const uint64_t d = bases32(q.words, q.base_off[qi] + static_cast<uint64_t>(x)) ^
                         target_bases32(idx.twords, idx.tbase[slot], len, qdi & 1,
                                        static_cast<int32_t>(x));
      differ = (b1 - x < 32 ? d >> (64 - 2 * (b1 - x)) : d) != 0;
    }
  }
  return !__syncthreads_or(differ);
}

constexpr int kProbeBlock = 256;

// One thread per window, blocks of whole 32-window tiles, `rounds` block widths of
// windows a block: the table probe (or the index's record of the window), then
// the run starts in the window's bucket.  Bound by latency: a chain of loads
// (the block's query, its target, bases, then a table slot and neighbours, all
// scattered, for a query that is no target of the index).  All HiFi reads (200
// million windows of indexed queries): 8.4 ms with a table probe and neighbours
// for each window, 2.2 with the records; 30 million windows of reads with 8 %
// errors: 1.95 ms, 1.55 with the index's filter.
__global__ void __launch_bounds__(kProbeBlock, 6) probe_kernel(
    DeviceIndex idx, QueryBatch q, int rounds, uint4* __restrict__ recs,
    uint32_t* __restrict__ nstart, uint32_t* __restrict__ cbits, uint32_t* __restrict__ fbits,
    uint32_t* __restrict__ tile_filt, uint32_t* __restrict__ tile_start) {
  __shared__ uint32_t ends[2];             // queries of the block's first and last windows
  __shared__ bool solid[kProbeBlock + 1];  // of the windows before and in the block
  const uint64_t w0 = static_cast<uint64_t>(blockIdx.x) * kProbeBlock * rounds;
  const uint64_t w1 = min(w0 + static_cast<uint64_t>(kProbeBlock) * rounds, q.nwin);
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 64) {
    const uint32_t e = query_of_warp(q.win_off, q.nq, threadIdx.x < 32 ? w0 : w1 - 1);
    if (lane == 0) ends[threadIdx.x >> 5] = e;
  }
  __syncthreads();
  uint32_t lo = ends[0];
  const bool indexed = ends[0] == ends[1] && indexed_windows(idx, q, lo, w0, w1);
  const uint4* row = nullptr;  // records of the query's target
  int64_t last = 0;            // the target's last window, for a query that is its reverse
  bool back = false;
  if (indexed) {
    const int32_t qdi = q.qdi[lo];
    row = idx.windows + idx.win_off[static_cast<uint32_t>(qdi) >> 1];
    last = static_cast<int64_t>(idx.slot_len[static_cast<uint32_t>(qdi) >> 1]) - idx.k;
    back = qdi & 1;
  }
  const uint64_t q0 = q.win_off[lo];
  for (uint64_t b0 = w0; b0 < w1; b0 += kProbeBlock) {
    const uint64_t w = b0 + threadIdx.x;
    uint64_t meta = 0, p = 0;
    uint32_t self = kNoSelf, left = 7;
    BucketSide side{7, 0};
    uint8_t fl = 0;
    if (w < w1 && indexed) {
      p = w - q0;
      const uint4* at = row + (back ? last - static_cast<int64_t>(p) : static_cast<int64_t>(p));
      const uint4 rec = __ldg(at);
      meta = static_cast<uint64_t>(rec.y) << 32 | rec.x;
      const bool rev = ((rec.w & kWindowRev) != 0) != back;
      if (rev) fl = kWinRev;
      if (rec.w & kWindowFound) {
        if (meta & kRepetitiveBit) {
          fl |= kWinFiltered;
        } else {
          fl |= kWinSolid;
          self = rec.z & kPlaceMask;
          side = record_side(rec, rev);
          if (p > 0) left = back ? 3u - (rec.z >> 30) : rec.z >> 28 & 3u;
        }
      }
      if (threadIdx.x == 0 && b0 == w0) {
        const uint4 r = p > 0 ? __ldg(at + (back ? 1 : -1)) : make_uint4(0, 0, 0, 0);
        solid[0] = (r.w & kWindowFound) && !(r.y >> 31);
      }
    } else if (w < w1) {
      uint32_t hi = ends[1];  // most blocks lie within one query
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(q.win_off + mid) <= w)
          lo = mid;
        else
          hi = mid - 1;
      }
      p = w - q.win_off[lo];
      fl = probe_run_window(idx, q, lo, p, meta, self, side);
      if (p > 0) left = base_at(q.words, q.base_off[lo] + p - 1);
      if (threadIdx.x == 0 && b0 == w0) {
        // the last window of the block before: could a run continue from it?
        bool before = false;
        if (p > 0) {
          uint64_t m;
          uint32_t a;
          BucketSide b;
          before = probe_run_window(idx, q, lo, p - 1, m, a, b) & kWinSolid;
        }
        solid[0] = before;
      }
    }
    solid[threadIdx.x + 1] = fl & kWinSolid;
    __syncthreads();
    const bool continues = solid[threadIdx.x];
    uint32_t ns = 0;
    RunTest rt{7, (fl & kWinRev) ? 4 : 0};
    if (fl & kWinSolid) {
      if (left != 7 && continues) rt.expect = rt.shift ? 3u - left : left;
      const uint64_t off = meta & kOffsetMask;
      const uint32_t c = bucket_size(meta), own = self != kNoSelf ? 1u : 0u;
      if (side.most != 7 && side.most != rt.expect && side.others == 0) rt.expect = 7;
      if (rt.expect == 7) {
        ns = c - own;
      } else {
        ns = side.most == rt.expect ? side.others : count_starts(idx, off, c, rt);
        // the query's own position is no hit
        if (!indexed && ns && own && own_before(idx, q.qdi[lo], p) != left) --ns;
      }
    }
    const uint32_t cb = __ballot_sync(0xffffffffu, fl & kWinSolid);
    const uint32_t fb = __ballot_sync(0xffffffffu, fl & kWinFiltered);
    const uint32_t starts = __reduce_add_sync(0xffffffffu, ns);
    if (w < w1) {
      nstart[w] = ns;
      if (ns || (fl & kWinFiltered))
        recs[w] = make_uint4(static_cast<uint32_t>(meta), static_cast<uint32_t>(meta >> 32),
                             static_cast<uint32_t>(p),
                             self | rt.expect << 22 | static_cast<uint32_t>(rt.shift) << 23);
      if (lane == 0) {
        cbits[w >> 5] = cb;
        fbits[w >> 5] = fb;
        tile_filt[w >> 5] = __popc(fb);
        tile_start[w >> 5] = starts;
      }
    }
    __syncthreads();  // solid is read
    if (threadIdx.x == kProbeBlock - 1) solid[0] = fl & kWinSolid;
  }
}

// First run and first filtered position of each query; in totals the most runs
// of a query, all runs, all filtered positions, and the number of queries in
// list: those that the large form of the sort takes.
__global__ void query_offsets_kernel(QueryBatch q, const uint32_t* __restrict__ nstart,
                                     const uint64_t* __restrict__ tile_off,
                                     const uint32_t* __restrict__ fbits,
                                     const uint64_t* __restrict__ ftile_off,
                                     uint64_t* __restrict__ q_off, uint64_t* __restrict__ f_off,
                                     unsigned long long* __restrict__ totals,
                                     uint32_t* __restrict__ list) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  auto first_run = [&](uint64_t w) {
    uint64_t o = tile_off[w >> 5];
    for (uint64_t j = w & ~31ull; j < w; ++j) o += nstart[j];  // inside a tile
    return o;
  };
  uint64_t o = 0;
  if (i <= q.nq) {
    const uint64_t w = q.win_off[i], t = w >> 5;
    const uint32_t r = static_cast<uint32_t>(w & 31);
    o = first_run(w);
    q_off[i] = o;
    const uint64_t f = ftile_off[t] + (r ? __popc(fbits[t] & ((1u << r) - 1u)) : 0);
    f_off[i] = f;
    if (i == q.nq) {
      totals[1] = o;
      totals[2] = f;
    }
  }
  uint64_t next = __shfl_down_sync(0xffffffffu, o, 1);
  if ((threadIdx.x & 31) == 31 && i < q.nq) next = first_run(q.win_off[i + 1]);
  uint32_t n = i < q.nq ? static_cast<uint32_t>(next - o) : 0u;
  if (n > kRunSortCap && n <= kRunSortLarge) list[atomicAdd(totals + 3, 1ull)] = i;
  n = __reduce_max_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0 && n) atomicMax(totals, static_cast<unsigned long long>(n));
}

// Which of 16 entries' nibbles differ from the pattern, entry i at bit i.
__device__ __forceinline__ uint32_t differ_bits16(uint4 x, int shift, uint32_t pat) {
  auto word = [&](uint32_t w) {  // one bit a byte, gathered by a multiplication
    const uint32_t d = ((((w >> shift) & 0x0f0f0f0fu) ^ pat) + 0x7f7f7f7fu) >> 7 & 0x01010101u;
    return d * 0x01020408u >> 24;  // bits 28 up are zero: the sums do not reach them
  };
  return word(x.x) | word(x.y) << 4 | word(x.z) << 8 | word(x.w) << 12;
}

// A warp writes its 32 windows' run starts.  The buckets of the windows that
// start runs (few windows do) are cut at every 16th entry; the pieces are
// numbered through and taken a lane each, which compares its 16 neighbour bytes
// at once, so the lanes are busy whether a bucket holds two entries or two
// hundred.  Bound by instructions and the scattered entries.
__global__ void __launch_bounds__(256) start_emit_kernel(
    DeviceIndex idx, QueryBatch q, const uint4* __restrict__ recs,
    const uint32_t* __restrict__ nstart, const uint64_t* __restrict__ tile_off,
    const uint32_t* __restrict__ fbits, const uint64_t* __restrict__ ftile_off,
    uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, int32_t* __restrict__ fpos) {
  const uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t ns = 0, fb = 0;
  if (w < q.nwin) {
    ns = nstart[w];
    fb = fbits[w >> 5];
  }
  const bool filtered = (fb >> lane) & 1u;
  uint4 rec = make_uint4(0, 0, 0, 0);
  if (ns || filtered) rec = recs[w];
  const uint32_t p = rec.z;
  if (filtered) fpos[ftile_off[w >> 5] + __popc(fb & lt)] = static_cast<int32_t>(p);
  if (!__any_sync(0xffffffffu, ns > 0)) return;
  const uint64_t meta = (static_cast<uint64_t>(rec.y) << 32) | rec.x, off = meta & kOffsetMask;
  const uint32_t test = rec.w, c = ns ? bucket_size(meta) : 0;
  const uint32_t pieces = ns ? (static_cast<uint32_t>(off & 15) + c + 15) >> 4 : 0;
  uint32_t upto = pieces;  // of this window and the ones before
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += y;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, upto, 31);
  uint64_t out = tile_off[w >> 5];
  for (uint32_t e0 = 0; e0 < total; e0 += 32) {
    const uint32_t j = e0 + lane;
    int src = 0;  // the window of piece j: the first whose count exceeds j
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (__shfl_sync(0xffffffffu, upto, src + o - 1) <= j) src += o;
    const uint32_t before = __shfl_sync(0xffffffffu, upto - pieces, src);
    const uint32_t n = __shfl_sync(0xffffffffu, c, src);
    const uint64_t wo = __shfl_sync(0xffffffffu, off, src);
    const uint32_t wp = __shfl_sync(0xffffffffu, p, src);
    const uint32_t wt = __shfl_sync(0xffffffffu, test, src);
    // the piece's 16 entries, the first of them (before the bucket's in its first piece)
    const int32_t first = static_cast<int32_t>((j - before) << 4) - static_cast<int32_t>(wo & 15);
    uint32_t m = 0;
    if (j < total) {
      const uint32_t expect = (wt >> 22) & 7u;
      m = expect == 7 ? 0xffffu
                      : differ_bits16(__ldg(reinterpret_cast<const uint4*>(idx.nbr) + (wo >> 4) +
                                            (j - before)),
                                      (wt >> 23) & 4u, expect * 0x01010101u);
      if (first < 0) m &= 0xffffu << -first;
      const int32_t end = static_cast<int32_t>(n) - first;  // entries of the bucket from here on
      if (end < 16) m &= (1u << end) - 1u;
      const uint32_t self = (wt & kNoSelf) - static_cast<uint32_t>(first);
      if (self < 16) m &= ~(1u << self);  // kNoSelf is beyond every bucket
    }
    uint32_t upto_m = __popc(m);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, upto_m, o);
      if (lane >= o) upto_m += y;
    }
    uint64_t d = out + upto_m - __popc(m);
    out += __shfl_sync(0xffffffffu, upto_m, 31);
    const uint64_t base = wo + static_cast<uint64_t>(static_cast<int64_t>(first));
    for (; m; m &= m - 1u, ++d) {
      const uint64_t sv = __ldg(idx.pos + base + (__ffs(m) - 1));
      uint32_t id = static_cast<uint32_t>(sv >> 32);
      int32_t pos = static_cast<int32_t>(sv & 0xffffffffu);
      if (wt >> 25) {
        pos = idx.slot_len[id >> 1] - pos - idx.k;
        id ^= 1u;
      }
      keys[d] = (static_cast<uint64_t>(id) << 32) | wp;
      vals[d] = static_cast<uint32_t>(pos);
    }
  }
}

// ---------------------------------------------------------------- sort, groups

template <int BLOCK, int ITEMS>
struct SortSmem {
  static constexpr int kCap = BLOCK * ITEMS;
  uint32_t id[kCap];
  uint16_t at[kCap];             // the run's place before the sort
  uint16_t wc[BLOCK / 32][256];  // per-warp digit counts, then offsets
  uint32_t dbase[256];
  uint32_t ws[8];
  uint32_t heads[BLOCK / 32];
  uint32_t item;
};
using SortSmall = SortSmem<512, 8>;
using SortLarge = SortSmem<1024, 16>;
static_assert(SortSmall::kCap == kRunSortCap && SortLarge::kCap == kRunSortLarge,
              "the sorts' capacities");

// A block a query: its runs (in cur-pos order) into (ext id, cur pos) order by a
// stable LSD radix sort of the ext ids, 8 bits a pass, and the number of its
// groups.  Ids and 16-bit places stay on chip; the runs themselves move once,
// where passes over device memory (match_radix, which queries beyond on_chip runs
// take beforehand) move them twice a digit and launch three kernels for it.  The
// small form takes all queries but the listed ones (of more than kRunSortCap and
// at most kRunSortLarge runs), which the large form takes when on_chip says so.
// One query of 5000 runs: 60 -> 30 us.
template <int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK, BLOCK > 512 ? 1 : 2)
    sort_queries_kernel(const uint64_t* __restrict__ q_off, uint32_t nq, uint32_t on_chip,
                        const uint32_t* __restrict__ list,
                        const unsigned long long* __restrict__ list_count, uint64_t* keys,
                        uint32_t* vals, int id_bits, uint32_t* __restrict__ q_groups,
                        uint32_t* __restrict__ work) {
  constexpr int kWarps = BLOCK / 32;
  constexpr bool kLarge = BLOCK > 512;
  extern __shared__ __align__(16) unsigned char sort_raw[];
  auto& sm = *reinterpret_cast<SortSmem<BLOCK, ITEMS>*>(sort_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t items = kLarge ? static_cast<uint32_t>(*list_count) : nq;
  for (;;) {
    if (threadIdx.x == 0) sm.item = atomicAdd(work, 1u);
    __syncthreads();
    const uint32_t item = sm.item;
    __syncthreads();
    if (item >= items) break;
    const uint32_t q = kLarge ? list[item] : item;
    if (kLarge && q >= nq) continue;  // the pass was cut after the list was made
    const uint64_t b = q_off[q];
    const uint64_t len = q_off[q + 1] - b;
    if (!kLarge && len > kRunSortCap && len <= on_chip) continue;
    const bool whole = len <= SortSmem<BLOCK, ITEMS>::kCap;
    const uint32_t n = whole ? static_cast<uint32_t>(len) : 0u;
    // warp w owns per_warp consecutive runs
    const uint32_t per_warp = ((n + BLOCK - 1) / BLOCK) * 32;
    const int rounds = static_cast<int>(per_warp / 32);
    const uint32_t j0 = warp * per_warp + lane;
    uint32_t id[ITEMS], at[ITEMS];  // at: the place, and in a pass the rank above it
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const uint32_t j = j0 + r * 32;
      id[r] = r < rounds && j < n ? static_cast<uint32_t>(keys[b + j] >> 32) : 0u;
      at[r] = j;
    }
    for (int shift = 0; n > 1 && shift < id_bits; shift += 8) {
      uint32_t* wc32 = reinterpret_cast<uint32_t*>(&sm.wc[0][0]);
      for (int i = threadIdx.x; i < kWarps * 128; i += BLOCK) wc32[i] = 0;
      __syncthreads();
#pragma unroll
      for (int r = 0; r < ITEMS; ++r) {
        if (r >= rounds) break;
        const bool in = j0 + r * 32 < n;
        const uint32_t d = in ? (id[r] >> shift) & 0xffu : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (in && lane == leader) {
          base = sm.wc[warp][d];
          sm.wc[warp][d] = static_cast<uint16_t>(base + __popc(peers));
        }
        base = __shfl_sync(0xffffffffu, base, leader);
        at[r] |= (base + __popc(peers & lt)) << 16;
        __syncwarp();
      }
      __syncthreads();
      uint32_t tot = 0, inc = 0;
      if (threadIdx.x < 256) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          const uint32_t c = sm.wc[w][threadIdx.x];
          sm.wc[w][threadIdx.x] = static_cast<uint16_t>(tot);
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
      for (int r = 0; r < ITEMS; ++r) {
        if (r < rounds && j0 + r * 32 < n) {
          const uint32_t d = (id[r] >> shift) & 0xffu;
          const uint32_t o = sm.dbase[d] + sm.wc[warp][d] + (at[r] >> 16);
          sm.id[o] = id[r];
          sm.at[o] = static_cast<uint16_t>(at[r]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < ITEMS; ++r) {
        const uint32_t j = j0 + r * 32;
        if (r < rounds && j < n) {
          id[r] = sm.id[j];
          at[r] = sm.at[j];
        }
      }
    }
    // in order now; longer queries are so in device memory.  Every run is read
    // before any is written
    uint32_t heads = n == 1 && threadIdx.x == 0;
    if (n > 1) {
      uint32_t x[ITEMS];
#pragma unroll
      for (int r = 0; r < ITEMS; ++r)
        if (r < rounds && j0 + r * 32 < n) x[r] = vals[b + at[r]];
      __syncthreads();
#pragma unroll
      for (int r = 0; r < ITEMS; ++r)
        if (r < rounds && j0 + r * 32 < n) vals[b + j0 + r * 32] = x[r];
#pragma unroll
      for (int r = 0; r < ITEMS; ++r)
        if (r < rounds && j0 + r * 32 < n) x[r] = static_cast<uint32_t>(keys[b + at[r]]);
      __syncthreads();
#pragma unroll
      for (int r = 0; r < ITEMS; ++r) {
        const uint32_t j = j0 + r * 32;
        if (r < rounds && j < n) {
          keys[b + j] = static_cast<uint64_t>(id[r]) << 32 | x[r];
          heads += j == 0 || id[r] != sm.id[j - 1];
        }
      }
    } else if (!whole) {
      for (uint64_t j = threadIdx.x; j < len; j += BLOCK)
        heads += j == 0 || (keys[b + j] >> 32) != (keys[b + j - 1] >> 32);
    }
    heads = __reduce_add_sync(0xffffffffu, heads);
    if (lane == 0) sm.heads[warp] = heads;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t g = 0;
      for (int w = 0; w < kWarps; ++w) g += sm.heads[w];
      q_groups[q] = g;
    }
  }
}

// The groups of each query: runs of one ext id among its sorted runs.  Bound by
// the latency of its steps, so a step takes eight runs a thread (59e6 runs in
// 3583 queries: 450 us with one, 255 with eight).
constexpr int kBoundItems = 8;

__global__ void __launch_bounds__(256) bounds_kernel(const uint64_t* __restrict__ q_off,
                                                     uint32_t nq,
                                                     const uint64_t* __restrict__ keys,
                                                     const uint64_t* __restrict__ q_group,
                                                     GroupInfo* __restrict__ bounds) {
  __shared__ uint32_t wsum[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (uint32_t q = blockIdx.x; q < nq; q += gridDim.x) {
    const uint64_t b = q_off[q], n = q_off[q + 1] - b;
    uint64_t g = q_group[q];
    int side = 0;
    for (uint64_t t0 = 0; t0 < n; t0 += 256 * kBoundItems, side ^= 1) {
      // a warp's runs are consecutive
      const uint64_t j0 = t0 + warp * (32 * kBoundItems) + lane;
      uint32_t id[kBoundItems];
      unsigned head[kBoundItems];
      uint32_t mine = 0;
#pragma unroll
      for (int r = 0; r < kBoundItems; ++r) {
        const uint64_t j = j0 + 32 * r;
        id[r] = j < n ? static_cast<uint32_t>(keys[b + j] >> 32) : 0u;
      }
#pragma unroll
      for (int r = 0; r < kBoundItems; ++r) {
        const uint64_t j = j0 + 32 * r;
        uint32_t prev = __shfl_up_sync(0xffffffffu, id[r], 1);
        if (lane == 0 && j > 0 && j < n) prev = static_cast<uint32_t>(keys[b + j - 1] >> 32);
        head[r] = __ballot_sync(0xffffffffu, j < n && (j == 0 || id[r] != prev));
        mine += __popc(head[r]);
      }
      if (lane == 0) wsum[side][warp] = mine;
      __syncthreads();
      uint32_t before = 0, all = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        before += w < warp ? wsum[side][w] : 0u;
        all += wsum[side][w];
      }
#pragma unroll
      for (int r = 0; r < kBoundItems; ++r) {
        if (head[r] >> lane & 1u) {
          GroupInfo gi{};
          gi.start = b + j0 + 32 * r;
          gi.query = q;
          gi.ext_di = id[r];
          bounds[g + before + __popc(head[r] & lt)] = gi;
        }
        before += __popc(head[r]);
      }
      g += all;
    }
    __syncthreads();  // wsum is free for the next query
  }
}

// Agreement of query and target over the next 32 bases from base k of a
// window on (m windows into a run): bases that agree, and the query's
// consecutive solid windows from the next one on, 32 at most.
__device__ __forceinline__ int32_t agree(uint64_t qb, uint64_t tb, uint32_t solid_bits) {
  const uint64_t diff = qb ^ tb;
  const int32_t same = diff ? __clzll(static_cast<long long>(diff)) >> 1 : 32;
  const uint32_t holes = ~solid_bits;
  return min(same, holes ? __ffs(holes) - 1 : 32);
}

constexpr int32_t kLongRoom = 96;    // room from which a run's end is looked for from there
constexpr int32_t kBack = 24;        // windows before the expected end

// Hits of the run that starts at window p of a query (first base qbase, first
// window w0) and position pos of a target strand: the windows over which the
// two agree, up to most, and up to the query's next window that is not solid.
// The first 32 bases alone decide most runs of noisy reads.
//
// room: windows from this run's first to the first of the group's next run (or
// up to the end of query or target when there is none).  No run starts between,
// so the hits of this run's diagonal in there are this run's, one after the
// other: a window of it that is a hit has nothing but hits before it.  A run
// usually ends k windows before the next one starts (or at the sequences' end),
// so one that outlasts its first 32 bases is taken up shortly before that place
// if the window there is a hit: the loads of a long run, which the warp's other
// lanes wait for, do not grow with its length (runs of 200 hits: all groups of
// all HiFi reads 7.4 -> 4.0 ms, against 64 bases a step all the way).
__device__ __forceinline__ int32_t run_length(const RunTables& t, uint64_t qbase, uint64_t w0,
                                              uint64_t tbase, int32_t tlen, bool rev, int32_t p,
                                              int32_t pos, int32_t most, int32_t room) {
  const int32_t k = t.idx.k;
  auto target32 = [&](int32_t x) {
    return target_bases32(t.idx.twords, tbase, tlen, rev, x);
  };
  int32_t m = 0;  // agreeing bases after the first window
  while (m < most - 1) {
    const uint64_t q0 = qbase + static_cast<uint64_t>(p) + k + m;
    const uint64_t b = w0 + static_cast<uint64_t>(p) + 1 + m;  // the next window
    const uint32_t bs = static_cast<uint32_t>(b & 31);
    const uint32_t c0 = __ldg(t.cbits + (b >> 5));
    const uint32_t c1 = bs ? __ldg(t.cbits + (b >> 5) + 1) : 0u;
    const int32_t step =
        agree(bases32(t.qb.words, q0), target32(pos + k + m), __funnelshift_r(c0, c1, bs));
    m += step;
    if (step < 32) break;
    if (m == 32 && room > kLongRoom) {
      const int32_t m0 = (room < most ? room - k : most) - kBack;
      const uint64_t d =
          bases32(t.qb.words, qbase + static_cast<uint64_t>(p) + m0) ^ target32(pos + m0);
      const uint64_t h = w0 + static_cast<uint64_t>(p) + m0;
      const bool solid = __ldg(t.cbits + (h >> 5)) >> (h & 31) & 1u;
      if (solid && (d >> (64 - 2 * k)) == 0) m = m0;
    }
  }
  return min(m + 1, most);
}

// Pieces of a group whose n runs (a, b, l by lane, from run i on) follow one
// another along its axis: slot piece0 holds element 0, the next slot the rest
// of its run, then one run a slot.
__device__ __forceinline__ void store_run_piece(const RunTables& t, uint64_t slot, uint32_t i,
                                                int32_t a, int32_t b, int32_t l) {
  if (i == 0) {
    // (the first slot goes unused when the first run is element 0 alone)
    t.pa[slot] = a;
    t.pb[slot] = b;
    t.pl[slot] = 1;
    const int32_t rest = l > 1 ? 1 : 0;
    t.pa[slot + 1] = a + rest;
    t.pb[slot + 1] = b + rest;
    t.pl[slot + 1] = l - rest;
  } else {
    t.pa[slot + 1 + i] = a;
    t.pb[slot + 1 + i] = b;
    t.pl[slot + 1 + i] = l;
  }
}

constexpr int kGroupWarps = 8;

// A warp a group.  Warps take chunks of consecutive groups from a counter and
// list a chunk's survivors with one counter update a list.  A warp's lanes
// wait for its longest run, and the loads of a step are scattered: four blocks
// an SM (64 registers; at five the spills cost more than the warps gain).  All
// groups of all HiFi reads (36e6 runs of 200 hits): 3.3 ms, at 0.7 instructions
// a cycle; 2.7e5 groups of 218 runs of 8 hits: 1.4 ms.
__global__ void __launch_bounds__(kGroupWarps * 32, 4) run_groups_kernel(RunTables t, ChainParams p,
                                                                      uint32_t chunk,
                                                                      uint32_t* work) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint64_t G = *t.ngroups;
  constexpr uint32_t kNone = kRunClasses + 2;
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(work, chunk);
    const uint64_t g0 = __shfl_sync(0xffffffffu, item, 0);
    if (g0 >= G) break;
    const uint32_t m = static_cast<uint32_t>(min(static_cast<uint64_t>(chunk), G - g0));
    uint32_t cls = kNone;  // of group g0 + lane
    bool ext = false;
    for (uint32_t u = 0; u < m; ++u) {
      const uint64_t g = g0 + u;
      const GroupInfo gi = t.bounds[g];
      const uint64_t end = g + 1 < G ? t.bounds[g + 1].start : t.nruns;
      const uint32_t n = static_cast<uint32_t>(end - gi.start);
      const uint32_t slot = gi.ext_di >> 1;
      const bool rev = gi.ext_di & 1u;
      const int32_t tlen = t.idx.slot_len[slot];
      const uint64_t tbase = t.idx.tbase[slot];
      const uint64_t qbase = t.qb.base_off[gi.query];
      const uint64_t w0 = t.qb.win_off[gi.query];
      const int32_t qwin = static_cast<int32_t>(t.qb.win_off[gi.query + 1] - w0);
      const int32_t cur_len = t.qinfo[gi.query].len;
      const bool es = tlen > cur_len;
      const uint64_t pslot = gi.start + g;
      uint32_t hits = 0, distinct = 0;
      int32_t mn = INT_MAX, mx = INT_MIN, first_c = 0, first_l = 0;
      int32_t end_c = 0, end_e = 0;  // ends of the runs so far (cur: greatest; ext: the last one's)
      bool ties = false, rising = true;
      for (uint32_t i0 = 0; i0 < n; i0 += 32) {
        const uint32_t i = i0 + lane;
        const bool in = i < n;
        int32_t c = 0, e = 0, l = 0;
        if (in) {
          c = static_cast<int32_t>(t.keys[gi.start + i] & 0xffffffffu);
          e = static_cast<int32_t>(t.vals[gi.start + i]);
          const int32_t most = min(qwin - c, tlen - t.idx.k + 1 - e);
          const int32_t room =
              i + 1 < n ? min(static_cast<int32_t>(t.keys[gi.start + i + 1] & 0xffffffffu) - c, most)
                        : most;
          l = run_length(t, qbase, w0, tbase, tlen, rev, c, e,
                         most, room);
          t.rlen[gi.start + i] = static_cast<uint32_t>(l);
          store_run_piece(t, pslot, i, es ? e : c, es ? c : e, l);
          hits += l;
          mn = min(mn, e);
          mx = max(mx, e + l - 1);
        }
        __syncwarp();
        if (i0 == 0) {
          first_c = __shfl_sync(0xffffffffu, c, 0);
          first_l = __shfl_sync(0xffffffffu, l, 0);
        }
        // greatest end of the runs before this one, and the last one's ext end
        int32_t inc = in ? c + l : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int32_t y = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc = max(inc, y);
        }
        int32_t before = __shfl_up_sync(0xffffffffu, inc, 1);
        before = lane == 0 ? end_c : max(before, end_c);
        int32_t pe = __shfl_up_sync(0xffffffffu, e + l, 1);
        if (lane == 0) pe = end_e;
        if (in) {
          distinct += max(0, c + l - max(c, before));
          ties |= c < before;
          rising &= e >= pe;
        }
        end_c = max(end_c, __shfl_sync(0xffffffffu, inc, 31));
        end_e = __shfl_sync(0xffffffffu, e + l, 31);  // used when more runs follow
      }
      hits = __reduce_add_sync(0xffffffffu, hits);
      distinct = __reduce_add_sync(0xffffffffu, distinct);
      mn = __reduce_min_sync(0xffffffffu, mn);
      mx = __reduce_max_sync(0xffffffffu, mx);
      ties = __any_sync(0xffffffffu, ties);
      rising = __all_sync(0xffffffffu, rising);
      const uint32_t uniq = distinct - (first_c == 0 ? 1u : 0u);
      if (prefilter_keeps(uniq, first_c, end_c - 1, mn, mx, cur_len, tlen, p)) {
        const bool ready = es ? rising : !ties;
        RunGroup rg{};
        rg.run0 = gi.start;
        rg.nruns = n;
        rg.piece0 = pslot + (first_l > 1 ? 0u : 1u);
        rg.npieces = n + (first_l > 1 ? 1u : 0u);
        rg.nhits = hits;
        rg.query = gi.query;
        rg.ext_di = gi.ext_di;
        rg.ext_len = tlen;
        rg.flags = (es ? kRunExt : 0u) | (ties ? kRunCurTies : 0u);
        if (lane == 0) t.groups[g] = rg;
        if (lane == static_cast<int>(u)) {
          cls = ready ? static_cast<uint32_t>(run_class(rg.npieces))
                      : kRunClasses + (n <= 32 ? 0u : 1u);
          ext = es;
        }
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < kNone; ++k) {
      const unsigned b = __ballot_sync(0xffffffffu, cls == k);
      if (!b) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(t.counts + kRcList + k, __popc(b));
      at = __shfl_sync(0xffffffffu, at, 0);
      uint32_t* list = k < kRunClasses ? t.lists + k * t.max_groups
                                       : t.sort_lists + (k - kRunClasses) * t.max_groups;
      if (cls == k) list[at + __popc(b & lt)] = static_cast<uint32_t>(g0) + lane;
    }
    const unsigned eb = __ballot_sync(0xffffffffu, ext);
    if (lane == 0 && eb) atomicAdd(t.counts + kRcExt, __popc(eb));
  }
}

// ---------------------------------------------------------------- open groups

__global__ void open_info_kernel(RunTables t, uint32_t nopen, OpenInfo* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nopen) return;
  const uint32_t g = t.open_list[i];
  const RunGroup& rg = t.groups[g];
  out[i] = OpenInfo{g, rg.query, rg.nhits, rg.flags};
}

// Cur positions that hits of an open group share, as (sub-batch query, key):
// where a run (in cur order) starts before the greatest end of the ones before.
__global__ void tie_keys_kernel(RunTables t, OpenBatch o, uint64_t* __restrict__ tie_q,
                                uint64_t* __restrict__ tie_key,
                                unsigned long long* __restrict__ count, uint64_t cap) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= o.n || o.src_q[i] == kNoLink) return;
  const RunGroup rg = t.groups[o.list[i]];
  uint32_t end = 0;  // greatest end of the runs so far
  for (uint32_t r0 = 0; r0 < rg.nruns; r0 += 32) {
    const uint32_t r = r0 + lane;
    const bool in = r < rg.nruns;
    const uint64_t key = in ? t.keys[rg.run0 + r] : 0;
    const uint32_t c = static_cast<uint32_t>(key), e = in ? c + t.rlen[rg.run0 + r] : 0u;
    uint32_t most = e;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, most, d);
      if (lane >= d) most = max(most, y);
    }
    uint32_t before = __shfl_up_sync(0xffffffffu, most, 1);
    before = lane == 0 ? end : max(before, end);
    const uint32_t n = in && min(e, before) > c ? min(e, before) - c : 0u;
    uint32_t upto = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, upto, 31);
    unsigned long long at = 0;
    if (lane == 0 && total) at = atomicAdd(count, static_cast<unsigned long long>(total));
    at = __shfl_sync(0xffffffffu, at, 0) + upto - n;
    for (uint32_t x = 0; x < n && at + x < cap; ++x) {
      tie_q[at + x] = o.src_q[i];
      tie_key[at + x] = key + x;
    }
    end = max(end, __shfl_sync(0xffffffffu, most, 31));
  }
}

// The open groups' hits in KmerMatch order: from their runs, or (groups that
// repeat a cur position) from their query's sorted hits.  kExpandSlices warps
// share a group: few groups are open, some of them long.
constexpr uint32_t kExpandSlices = 16;

__global__ void expand_kernel(RunTables t, OpenBatch o, uint64_t* __restrict__ keys,
                              uint32_t* __restrict__ vals, GroupInfo* __restrict__ groups,
                              uint32_t* __restrict__ ext_list, uint32_t* __restrict__ dp_list,
                              uint32_t* __restrict__ counts) {
  const int lane = threadIdx.x & 31;
  const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t li = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; li < o.n; li += nwarps) {
    const RunGroup rg = t.groups[o.list[li]];
    const uint32_t slice = blockIdx.y;
    uint64_t d = o.off[li];
    if (lane == 0 && slice == 0) {
      GroupInfo gi{};
      gi.start = d;
      gi.n = rg.nhits;
      gi.query = rg.query;
      gi.ext_di = rg.ext_di;
      gi.ext_len = rg.ext_len;
      gi.survive = 1;
      gi.ext_sorted = (rg.flags & kRunExt) ? 1 : 0;
      groups[li] = gi;
      dp_list[atomicAdd(counts + 1, 1u)] = li;
      if (gi.ext_sorted) ext_list[atomicAdd(counts + 0, 1u)] = li;
    }
    const uint32_t sq = o.src_q[li];
    if (sq != kNoLink) {
      uint64_t lo = o.sorted_off[sq], hi = o.sorted_off[sq + 1];
      const uint64_t end = hi, first = static_cast<uint64_t>(rg.ext_di) << 32;
      while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (o.sorted_keys[mid] < first)
          lo = mid + 1;
        else
          hi = mid;
      }
      for (uint32_t j = slice * 32 + lane; j < rg.nhits && lo + j < end;
           j += 32 * kExpandSlices) {
        keys[d + j] = o.sorted_keys[lo + j];
        vals[d + j] = o.sorted_vals[lo + j];
      }
      continue;
    }
    for (uint32_t i0 = 0; i0 < rg.nruns; i0 += 32) {
      const uint32_t i = i0 + lane, n = min(32u, rg.nruns - i0);
      const uint32_t len = lane < static_cast<int>(n) ? t.rlen[rg.run0 + i] : 0u;
      if (i0 / 32 % kExpandSlices != slice) {
        d += __reduce_add_sync(0xffffffffu, len);
        continue;
      }
      const uint64_t first = lane < static_cast<int>(n) ? t.keys[rg.run0 + i] : 0;
      const uint32_t ext = lane < static_cast<int>(n) ? t.vals[rg.run0 + i] : 0u;
      for (uint32_t r = 0; r < n; ++r) {
        const uint64_t key = __shfl_sync(0xffffffffu, first, r);
        const uint32_t e = __shfl_sync(0xffffffffu, ext, r), l = __shfl_sync(0xffffffffu, len, r);
        for (uint32_t j = lane; j < l; j += 32) {
          keys[d + j] = key + j;
          vals[d + j] = e + j;
        }
        d += l;
      }
    }
  }
}

// Rows of a batch of open groups join the pool under their run groups.
__global__ void append_rows_kernel(const OverlapRow* __restrict__ from,
                                   const uint32_t* __restrict__ nfrom,
                                   const uint32_t* __restrict__ list,
                                   OverlapRow* __restrict__ pool, uint64_t pool_cap,
                                   uint32_t* __restrict__ pool_count, DeviceStatus* st) {
  const uint32_t n = *nfrom;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    OverlapRow r = from[i];
    if (r.rank == kRankDropped) continue;
    r.group = list[r.group];
    const uint32_t d = atomicAdd(pool_count, 1u);
    if (d < pool_cap)
      pool[d] = r;
    else
      raise_status(st, kDevProposalOverflow, 1, static_cast<int64_t>(r.group));
  }
}

// A group that runs_settle_first listed and the run path then finished.
__device__ __forceinline__ bool settled(const RunGroup& g) {
  return g.first != 0 && !(g.flags & kRunOpen);
}

__global__ void settle_first_kernel(RunTables t, OpenBatch o, const uint64_t* __restrict__ keys,
                                    const uint32_t* __restrict__ vals,
                                    const GroupInfo* __restrict__ groups,
                                    uint32_t* __restrict__ lists, uint32_t* __restrict__ counts) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= o.n) return;
  RunGroup& g = t.groups[o.list[i]];
  if (!(g.flags & kRunFirst)) return;
  const GroupInfo gi = groups[i];
  int32_t cur = static_cast<int32_t>(keys[gi.start] & 0xffffffffu);
  int32_t ext = static_cast<int32_t>(vals[gi.start]);
  if (gi.ext_sorted == 1) {  // re-sorted: key ext pos, value cur pos
    const int32_t x = cur;
    cur = ext;
    ext = x;
  }
  const bool es = g.flags & kRunExt;
  const int32_t a = es ? ext : cur, b = es ? cur : ext;
  const uint32_t n = min(g.npieces, 32u);
  for (uint32_t z = 0; z < n && t.pa[g.piece0 + z] == a; ++z) {
    if (t.pb[g.piece0 + z] != b) continue;
    if (t.pl[g.piece0 + z] != 1) return;  // element 0 is a piece of its own
    g.first = z + 1;
    g.flags &= ~static_cast<uint32_t>(kRunOpen | kRunFirst);
    lists[atomicAdd(counts + kRcList, 1u)] = o.list[i];  // one class: all in the first list
    return;
  }
}

__global__ void unsettled_kernel(RunTables t, OpenBatch o, uint32_t* __restrict__ dp_list,
                                 uint32_t* __restrict__ count) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < o.n && !settled(t.groups[o.list[i]])) dp_list[atomicAdd(count, 1u)] = i;
}

__global__ void fold_rows_kernel(RunTables t, const uint32_t* __restrict__ open_list,
                                 uint32_t nopen, const uint32_t* __restrict__ rows,
                                 uint32_t* __restrict__ group_rows) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nopen && !settled(t.groups[open_list[i]])) group_rows[open_list[i]] = rows[i];
}

__global__ void scatter_rows_kernel(const OverlapRow* __restrict__ pool,
                                    const uint32_t* __restrict__ npool,
                                    const uint32_t* __restrict__ kept,
                                    const uint64_t* __restrict__ kept_off,
                                    OverlapRow* __restrict__ rows) {
  const uint32_t n = *npool;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const OverlapRow r = pool[i];
    if (r.rank < kept[r.group]) rows[kept_off[r.group] + r.rank] = r;
  }
}

}  // namespace

cudaError_t index_neighbours(const uint64_t* pos, uint64_t npos, const uint64_t* words,
                             const uint64_t* base_off, const int32_t* slot_len, int k,
                             uint8_t* nbr, cudaStream_t s) {
  if (npos == 0) return cudaSuccess;
  count_launch();
  neighbour_kernel<<<grid(npos, 256), 256, 0, s>>>(pos, npos, words, base_off, slot_len, k, nbr);
  return cudaGetLastError();
}

cudaError_t runs_count(const DeviceIndex& idx, const QueryBatch& q, uint4* recs, uint32_t* nstart,
                       uint32_t* cbits, uint32_t* fbits, uint32_t* tile_filt,
                       uint32_t* tile_start, int num_sms, cudaStream_t s) {
  if (q.nwin == 0) return cudaSuccess;
  // up to eight rounds a block, as long as the blocks fill the chip four times
  const int rounds = static_cast<int>(std::clamp<uint64_t>(
      q.nwin / (4ull * 6 * num_sms * kProbeBlock), 1, 8));
  count_launch();
  probe_kernel<<<grid(q.nwin, kProbeBlock * rounds), kProbeBlock, 0, s>>>(
      idx, q, rounds, recs, nstart, cbits, fbits, tile_filt, tile_start);
  return cudaGetLastError();
}

cudaError_t runs_query_offsets(const QueryBatch& q, const uint32_t* nstart,
                               const uint64_t* tile_off, const uint32_t* fbits,
                               const uint64_t* ftile_off, uint64_t* q_off, uint64_t* f_off,
                               unsigned long long* totals, uint32_t* list,
                               cudaStream_t s) {
  count_launch();
  query_offsets_kernel<<<grid(q.nq + 1ull, 128), 128, 0, s>>>(q, nstart, tile_off, fbits,
                                                              ftile_off, q_off, f_off, totals,
                                                              list);
  return cudaGetLastError();
}

cudaError_t runs_emit(const DeviceIndex& idx, const QueryBatch& q, const uint4* recs,
                      const uint32_t* nstart, const uint64_t* tile_off, const uint32_t* fbits,
                      const uint64_t* ftile_off, uint64_t* keys, uint32_t* vals, int32_t* fpos,
                      cudaStream_t s) {
  if (q.nwin == 0) return cudaSuccess;
  count_launch();
  start_emit_kernel<<<grid(q.nwin, 256), 256, 0, s>>>(idx, q, recs, nstart, tile_off, fbits,
                                                      ftile_off, keys, vals, fpos);
  return cudaGetLastError();
}

cudaError_t runs_sort(const uint64_t* q_off, uint32_t nq, uint64_t longest, uint32_t on_chip,
                      const uint32_t* list,
                      const unsigned long long* list_count, uint64_t* keys, uint32_t* vals,
                      int id_bits, uint32_t* q_groups, uint32_t* work, int num_sms,
                      cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  auto launch = [&](auto kernel, size_t smem, int block, int per_sm, uint32_t* counter) {
    const cudaError_t e = cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    count_launch();
    kernel<<<static_cast<unsigned>(std::min<uint64_t>(nq, static_cast<uint64_t>(per_sm) * num_sms)),
             block, smem, s>>>(q_off, nq, on_chip, list, list_count, keys, vals, id_bits, q_groups, counter);
    return cudaGetLastError();
  };
  cudaError_t e = cudaSuccess;
  if (longest > kRunSortCap && on_chip > kRunSortCap)
    e = launch(sort_queries_kernel<1024, 16>, sizeof(SortLarge), 1024, 1, work + 1);
  if (e == cudaSuccess) e = launch(sort_queries_kernel<512, 8>, sizeof(SortSmall), 512, 2, work);
  return e;
}

cudaError_t runs_bounds(const uint64_t* q_off, uint32_t nq, const uint64_t* keys,
                        const uint64_t* q_group, GroupInfo* bounds, int num_sms, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  count_launch();
  bounds_kernel<<<static_cast<unsigned>(std::min<uint64_t>(nq, 8ull * num_sms)), 256, 0, s>>>(
      q_off, nq, keys, q_group, bounds);
  return cudaGetLastError();
}

cudaError_t runs_groups(const RunTables& t, const ChainParams& p, int num_sms, cudaStream_t s) {
  if (t.max_groups == 0) return cudaSuccess;
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, run_groups_kernel,
                                                                kGroupWarps * 32, 0);
  if (e != cudaSuccess) return e;
  // chunks of up to 32 groups, at least eight a resident warp (few groups: one
  // each, so that they run side by side)
  const uint64_t warps = static_cast<uint64_t>(std::max(per_sm, 1)) * num_sms * kGroupWarps;
  const uint32_t chunk =
      static_cast<uint32_t>(std::min<uint64_t>(32, std::max<uint64_t>(1, t.max_groups / (8 * warps))));
  const uint64_t need = (t.max_groups + chunk - 1) / chunk;
  count_launch();
  run_groups_kernel<<<static_cast<unsigned>(std::min((need + kGroupWarps - 1) / kGroupWarps,
                                                     warps / kGroupWarps)),
                      kGroupWarps * 32, 0, s>>>(t, p, chunk, t.counts + kRcWork);
  return cudaGetLastError();
}

cudaError_t runs_open_info(const RunTables& t, uint32_t nopen, OpenInfo* out, cudaStream_t s) {
  if (nopen == 0) return cudaSuccess;
  count_launch();
  open_info_kernel<<<grid(nopen, 256), 256, 0, s>>>(t, nopen, out);
  return cudaGetLastError();
}

cudaError_t runs_tie_keys(const RunTables& t, const OpenBatch& o, uint64_t* tie_q,
                          uint64_t* tie_key, unsigned long long* count, uint64_t cap,
                          cudaStream_t s) {
  if (o.n == 0) return cudaSuccess;
  count_launch();
  tie_keys_kernel<<<grid(o.n * 32ull, 64), 64, 0, s>>>(t, o, tie_q, tie_key, count, cap);
  return cudaGetLastError();
}

cudaError_t runs_expand(const RunTables& t, const OpenBatch& o, uint64_t* keys, uint32_t* vals,
                        GroupInfo* groups, uint32_t* ext_list, uint32_t* dp_list,
                        uint32_t* counts, int num_sms, cudaStream_t s) {
  if (o.n == 0) return cudaSuccess;
  count_launch();
  const dim3 blocks(static_cast<unsigned>(std::min<uint64_t>(grid(o.n * 32ull, 256),
                                                             16ull * num_sms)),
                    kExpandSlices);
  expand_kernel<<<blocks, 256, 0, s>>>(t, o, keys, vals, groups, ext_list, dp_list, counts);
  return cudaGetLastError();
}

cudaError_t runs_append_rows(const OverlapRow* from, const uint32_t* nfrom, const uint32_t* list,
                             OverlapRow* pool, uint64_t pool_cap, uint32_t* pool_count,
                             DeviceStatus* st, int num_sms, cudaStream_t s) {
  count_launch();
  append_rows_kernel<<<num_sms, 256, 0, s>>>(from, nfrom, list, pool, pool_cap, pool_count, st);
  return cudaGetLastError();
}

cudaError_t runs_settle_first(const RunTables& t, const OpenBatch& o, const uint64_t* keys,
                              const uint32_t* vals, const GroupInfo* groups, uint32_t* lists,
                              uint32_t* counts, cudaStream_t s) {
  if (o.n == 0) return cudaSuccess;
  count_launch();
  settle_first_kernel<<<grid(o.n, 128), 128, 0, s>>>(t, o, keys, vals, groups, lists, counts);
  return cudaGetLastError();
}

cudaError_t runs_unsettled(const RunTables& t, const OpenBatch& o, uint32_t* dp_list,
                           uint32_t* count, cudaStream_t s) {
  if (o.n == 0) return cudaSuccess;
  count_launch();
  unsettled_kernel<<<grid(o.n, 128), 128, 0, s>>>(t, o, dp_list, count);
  return cudaGetLastError();
}

cudaError_t runs_fold_rows(const RunTables& t, const uint32_t* open_list, uint32_t nopen,
                           const uint32_t* rows, uint32_t* group_rows, cudaStream_t s) {
  if (nopen == 0) return cudaSuccess;
  count_launch();
  fold_rows_kernel<<<grid(nopen, 256), 256, 0, s>>>(t, open_list, nopen, rows, group_rows);
  return cudaGetLastError();
}

cudaError_t runs_scatter_rows(const OverlapRow* pool, const uint32_t* npool, uint64_t max_pool,
                              const uint32_t* kept, const uint64_t* kept_off, OverlapRow* rows,
                              cudaStream_t s) {
  if (max_pool == 0) return cudaSuccess;
  count_launch();
  scatter_rows_kernel<<<std::min(grid(max_pool, 256), 2048u), 256, 0, s>>>(pool, npool, kept,
                                                                          kept_off, rows);
  return cudaGetLastError();
}

}  // namespace cuflye
