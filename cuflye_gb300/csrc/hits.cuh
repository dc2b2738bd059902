// hits.cuh — one query window's table probe, shared by hit counting (hits.cu)
// and run counting (runs.cu).
#pragma once

#include <cstdint>

#include "common.cuh"
#include "kernels.h"

namespace cuflye {

__device__ __forceinline__ uint32_t query_of(const uint64_t* __restrict__ win_off, uint32_t nq,
                                             uint64_t w) {
  uint32_t lo = 0, hi = nq - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (__ldg(win_off + mid) <= w)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// The same by a whole warp, 32 candidates a step: three loads in a row where
// the halving search has thirteen (13 thousand queries).
__device__ __forceinline__ uint32_t query_of_warp(const uint64_t* __restrict__ win_off,
                                                  uint32_t nq, uint64_t w) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = 0, n = nq;  // the answer is in [lo, lo + n)
  while (n > 1) {
    const uint32_t step = (n + 31) / 32, at = lane * step;
    const unsigned m =
        __ballot_sync(0xffffffffu, at < n && __ldg(win_off + lo + at) <= w) | 1u;
    const uint32_t j = 31 - __clz(m);
    lo += j * step;
    n = min(step, n - j * step);
  }
  return lo;
}

// The table word of a standard form, if the index has it.
__device__ __forceinline__ uint64_t index_probe(const DeviceIndex& idx, uint64_t key,
                                                bool* found) {
  if (idx.filter) {
    const uint64_t h = mix64(key);
    const uint32_t bits = filter_bits(h);
    if ((__ldg(idx.filter + filter_word(h, idx.filter_mask)) & bits) != bits) {
      *found = false;
      return 0;
    }
  }
  return table_probe(idx.table, idx.cap, key, found);
}

struct WindowKmer {
  uint64_t x;    // forward k-mer (Kmer::numRepr)
  uint64_t key;  // standard form
  bool rev;      // x is not in standard form
};

__device__ __forceinline__ WindowKmer window_kmer(const QueryBatch& q, uint32_t qi, uint64_t p,
                                                  int k) {
  WindowKmer w;
  w.x = kmer_at(q.words, q.base_off[qi] + p, k);
  const uint64_t rc = revcomp(w.x, k);
  w.rev = rc < w.x;
  w.key = w.rev ? rc : w.x;
  return w;
}

// Where a query's own window would be stored: (dense id, position) of the
// entry that is the self hit, flipped when the lookup flips (~0: none).
__device__ __forceinline__ uint64_t self_entry(const DeviceIndex& idx, int32_t qdi, uint64_t p,
                                               bool rev) {
  if (!(idx.transform && rev)) return (static_cast<uint64_t>(qdi) << 32) | static_cast<uint32_t>(p);
  const uint32_t sid = static_cast<uint32_t>(qdi) ^ 1u;
  const int32_t slen = idx.slot_len[sid >> 1];
  const int64_t sp = static_cast<int64_t>(slen) - static_cast<int64_t>(p) - idx.k;
  return sp >= 0 ? ((static_cast<uint64_t>(sid) << 32) | static_cast<uint32_t>(sp)) : ~0ULL;
}

// Index of entry `want` in a built bucket of c entries (sorted by (stored id,
// stored position), entries unique), or c.
__device__ __forceinline__ uint32_t bucket_find(const DeviceIndex& idx, uint64_t off, uint32_t c,
                                                uint64_t want) {
  uint32_t lo = 0, hi = c;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(idx.pos + off + mid) < want)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < c && __ldg(idx.pos + off + lo) == want ? lo : c;
}

constexpr uint32_t kPlaceMask = (1u << kCountBits) - 1;

// Position of query window p on the forward strand of its target (dense id
// qdi); negative or past the target's last window when it is not one of them.
__device__ __forceinline__ int64_t forward_window(const DeviceIndex& idx, int32_t qdi,
                                                  uint64_t p) {
  const int64_t f = static_cast<int64_t>(p);
  return (qdi & 1) ? static_cast<int64_t>(idx.slot_len[static_cast<uint32_t>(qdi) >> 1]) - idx.k - f
                   : f;
}

// Whether the indexed sequence of dense id qdi has the query's k-mer x at the
// query's position p: its own position is an entry of x's bucket exactly then
// (a look at the packed target, in step with the query's own bases).  rec: the
// index's record of the target's window, if it keeps any (loaded beside the
// target's bases, not after the comparison).
__device__ __forceinline__ bool own_window(const DeviceIndex& idx, int32_t qdi, uint64_t p,
                                           uint64_t x, uint4& rec) {
  rec = make_uint4(0, 0, 0, 0);
  if (qdi < 0 || !idx.twords) return false;
  const uint32_t slot = static_cast<uint32_t>(qdi) >> 1;
  const int64_t f = forward_window(idx, qdi, p);
  if (f < 0 || f + idx.k > idx.slot_len[slot]) return false;
  if (idx.windows) rec = __ldg(idx.windows + idx.win_off[slot] + static_cast<uint64_t>(f));
  const uint64_t y = kmer_at(idx.twords, idx.tbase[slot] + static_cast<uint64_t>(f), idx.k);
  return ((qdi & 1) ? revcomp(y, idx.k) : y) == x;
}

// A window's bucket: its table meta, flags (kWinRev, kWinFiltered,
// kWinTrivial), hits (the bucket's entries less the query's own position) and
// the own entry's bucket index (kWinTrivial on a built index).
struct WindowProbe {
  uint64_t meta;
  uint32_t hits;
  uint32_t self;
  uint8_t flags;
};

__device__ __forceinline__ WindowProbe probe_window(const DeviceIndex& idx, const QueryBatch& q,
                                                    uint32_t qi, uint64_t p,
                                                    uint32_t* __restrict__ q_tie) {
  const WindowKmer km = window_kmer(q, qi, p, idx.k);
  uint4 rec;
  const bool recorded = own_window(idx, q.qdi[qi], p, km.x, rec) && idx.windows;
  bool found = rec.w & kWindowFound;
  const uint64_t meta = recorded ? static_cast<uint64_t>(rec.y) << 32 | rec.x
                                 : index_probe(idx, km.key, &found);
  uint32_t c = 0, self = 0;
  uint8_t fl = km.rev ? kWinRev : 0;
  if (found && (meta & kRepetitiveBit)) {
    fl |= kWinFiltered;
  } else if (found) {
    c = static_cast<uint32_t>((meta >> 40) & ((1ULL << kCountBits) - 1));
    if (q_tie && (meta & kDupIdsBit) && q_tie[qi] == 0) atomicOr(q_tie + qi, 1u);
    const int32_t qdi = q.qdi[qi];
    if (c > 0 && qdi >= 0) {
      // is the query's own window among the bucket entries?
      const uint64_t want = self_entry(idx, qdi, p, km.rev);
      const uint64_t off = meta & kOffsetMask;
      uint32_t self_hits = 0;
      if (idx.transform) {
        // built buckets are sorted by (stored id, stored position), entries
        // unique.  A query that is an indexed target finds its own entry
        // where the index recorded it (checked: a query sequence that
        // differs from the indexed one searches as any other)
        bool known = recorded;
        uint32_t at = rec.z & kPlaceMask;
        if (!known && idx.windows && !(qdi & 1)) {
          const uint32_t slot = static_cast<uint32_t>(qdi) >> 1;
          const uint64_t w0 = idx.win_off[slot];
          if (w0 + p < idx.win_off[slot + 1]) {
            at = idx.windows[w0 + p].z & kPlaceMask;
            known = at < c && __ldg(idx.pos + off + at) == want;
          }
        }
        if (!known) {
          at = bucket_find(idx, off, c, want);
          known = at < c;
        }
        self_hits = known ? 1u : 0u;
        if (self_hits) self = at;
      } else {
        // explicit entries keep input order and may repeat
        for (uint32_t e = 0; e < c; ++e) self_hits += __ldg(idx.pos + off + e) == want;
      }
      if (self_hits) {
        c -= self_hits;
        fl |= kWinTrivial;
      }
    }
  }
  return WindowProbe{meta, c, self, fl};
}

}  // namespace cuflye
