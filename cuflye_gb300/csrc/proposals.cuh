// proposals.cuh — overlap proposals of a target group: overlapTest and the
// k-mer divergence of one walked chain, and the group's primary selection
// (chain.cu walks hits, run_chain.cu runs).
#pragma once

#include <climits>
#include <cstdint>

#include "common.cuh"
#include "introsort.cuh"
#include "kernels.h"

namespace cuflye {

constexpr int kMaxProposals = kMaxGroupRows;

struct Prop {
  int32_t cb, ce, eb, ee, score, clen;
  float div;
};

__device__ __forceinline__ bool overlap_test(const Prop& o, int64_t cur_id, int64_t ext_id,
                                             int32_t cur_len, int32_t ext_len,
                                             const ChainParams& p) {
  const int32_t cr = o.ce - o.cb, er = o.ee - o.eb;
  if (cr < p.min_overlap || er < p.min_overlap) return false;
  const int32_t diff = abs(cr - er);
  if (static_cast<float>(diff) > fmul(0.5f, static_cast<float>(min(cr, er)))) return false;
  if (cur_id == ext_id) {
    const int32_t inter = min(o.ce, o.ee) - max(o.cb, o.eb);
    if (static_cast<float>(inter) > fdiv(static_cast<float>(cr), 2.0f)) return false;
  }
  if (cur_id == -ext_id) {
    const int32_t inter = min(o.ce, ext_len - o.eb) - max(o.cb, ext_len - o.ee);
    if (static_cast<float>(inter) > fdiv(static_cast<float>(cr), 2.0f)) return false;
  }
  if (!p.force_local && p.check_overhang) {
    const int32_t lr = max(min(o.cb, o.eb), min(cur_len - o.ce, ext_len - o.ee));
    if (lr > p.max_overhang) return false;
  }
  return true;
}

// First i in [0, n) with a[i] >= x (n: none), by the whole warp: 32 probes a
// round instead of one (a search of 167,000 entries waits for four loads, not
// seventeen).
template <class T>
__device__ __forceinline__ uint32_t warp_lower_bound(const T* __restrict__ a, uint32_t n, T x) {
  const int lane = threadIdx.x & 31;
  uint32_t lo = 0, hi = n;  // the answer lies in [lo, hi]
  while (lo < hi) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint32_t i = lo + static_cast<uint32_t>(lane) * step;  // (probes rise with the lane)
    const unsigned below = __ballot_sync(0xffffffffu, i < hi && __ldg(a + i) < x);
    // probes below x come first; the answer is past the last of them
    const uint32_t c = __popc(below);
    if (c == 0) return lo;
    hi = min(hi, lo + c * step);
    lo = lo + (c - 1) * step + 1;
  }
  return lo;
}

// Row ranks: a row whose divergence is still to be computed (its div holds the
// logarithm's argument), and a row that is over max_divergence.
constexpr uint32_t kRankOpen = 0x80000000u;
constexpr uint32_t kRankDropped = 0xffffffffu;

// overlapTest and the k-mer match rate of proposal o by the whole warp; a kept
// proposal is counted by every lane and appended to lane 0's props, its div
// holding 1 / rate: the divergence is the logarithm of that over k.
__device__ __forceinline__ void keep_proposal(Prop o, const QueryInfo& qi, int64_t ext_signed,
                                              int32_t ext_len, const int32_t* fq, uint32_t nf,
                                              const ChainParams& p,
                                              DeviceStatus* st, uint32_t gidx, Prop* props,
                                              int& np, bool& overflow) {
  bool keep = overlap_test(o, qi.signed_id, ext_signed, qi.len, ext_len, p);
  if (keep) {
    const uint32_t lo = warp_lower_bound(fq, nf, o.cb);
    const uint32_t hi = warp_lower_bound(fq, nf, o.ce + 1);
    const int32_t norm = max(o.ce - o.cb, o.ee - o.eb) - static_cast<int32_t>(hi - lo);
    keep = norm > 0;
    if (keep) {
      float rate = fdiv(fmul(static_cast<float>(o.clen), p.sample_rate), static_cast<float>(norm));
      rate = rate < 1.0f ? rate : 1.0f;
      const float x = fdiv(1.0f, rate);
      if (!(x < 16777216.0f)) raise_status(st, kDevLogDomain, 0, static_cast<int64_t>(gidx));
      o.div = x;
    }
  }
  if (keep) {
    if (np == kMaxProposals) {
      raise_status(st, kDevProposalOverflow, 0, static_cast<int64_t>(gidx));
      overflow = true;
    } else {
      if ((threadIdx.x & 31) == 0) props[np] = o;
      ++np;
    }
  }
}

// The group's proposals sorted by score descending in libstdc++ order, the
// primary ones kept under max_divergence, as rows in the pool.  One thread.
// A group's only row leaves its divergence to open_rows_kernel: the logarithm
// is a chain of double-precision operations, of which an SM does two a cycle,
// so a warp computes 32 rows' as fast as one.
__device__ __forceinline__ void finish_group(const Prop* props, int np, const QueryInfo& qi,
                                             uint32_t query, uint32_t ext_di, int32_t ext_len,
                                             uint32_t gidx, const LogfTable& logt,
                                             const ChainParams& p, OverlapRow* __restrict__ pool, uint64_t pool_cap,
                                             uint32_t* __restrict__ pool_count,
                                             uint32_t* __restrict__ group_rows,
                                             DeviceStatus* st) {
  if (np == 0) {
    group_rows[gidx] = 0;
    return;
  }
  // proposals by score descending, libstdc++ order
  uint64_t K[kMaxProposals];
  uint32_t V[kMaxProposals];
  for (int i = 0; i < np; ++i) {
    K[i] = static_cast<uint64_t>(static_cast<uint32_t>(INT_MAX - props[i].score));
    V[i] = static_cast<uint32_t>(i);
  }
  isort::serial_introsort(K, V, 0, static_cast<uint32_t>(np),
                          isort::depth_limit(static_cast<uint32_t>(np)));
  int prim[kMaxProposals];
  int nprim = 0;
  if (p.only_max_ext) {
    if (np > 0) prim[nprim++] = static_cast<int>(V[0]);
  } else {
    for (int s = 0; s < np; ++s) {
      const Prop& o = props[V[s]];
      bool contained = false;
      for (int t = 0; t < nprim && !contained; ++t) {
        const Prop& pr = props[prim[t]];
        contained = pr.cb <= o.cb && o.ce <= pr.ce && pr.eb <= o.eb && o.ee <= pr.ee &&
                    pr.score > o.score;
      }
      if (!contained) prim[nprim++] = static_cast<int>(V[s]);
    }
  }
  const bool one = nprim == 1;
  float div[kMaxProposals];
  int nk = 0;  // (prim is compacted in place)
  for (int t = 0; t < nprim; ++t) {
    const float x = props[prim[t]].div;
    const float d = one ? x : fdiv(flye_logf(x, logt), static_cast<float>(p.k));
    if (one || d < p.max_divergence) {
      prim[nk] = prim[t];
      div[nk++] = d;
    }
  }
  group_rows[gidx] = static_cast<uint32_t>(nk);
  if (nk == 0) return;
  const uint32_t base = atomicAdd(pool_count, static_cast<uint32_t>(nk));
  if (base + nk > pool_cap) {
    raise_status(st, kDevProposalOverflow, 1, static_cast<int64_t>(gidx));
    return;
  }
  for (int t = 0; t < nk; ++t) {
    const Prop& o = props[prim[t]];
    OverlapRow r;
    r.query = query;
    r.ext_di = ext_di;
    r.cur_begin = o.cb;
    r.cur_end = o.ce;
    r.cur_len = qi.len;
    r.ext_begin = o.eb;
    r.ext_end = o.ee;
    r.ext_len = ext_len;
    r.score = o.score;
    r.chain_len = o.clen;
    r.div = div[t];
    r.group = gidx;
    r.rank = static_cast<uint32_t>(t) | (one ? kRankOpen : 0u);
    pool[base + t] = r;
  }
}

}  // namespace cuflye
