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

constexpr int kMaxProposals = 64;

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

__device__ __forceinline__ uint32_t lower_bound_i32(const int32_t* a, uint32_t n, int32_t x) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// overlapTest, then the k-mer divergence of proposal o (its div is set here);
// kept proposals are appended to props.
__device__ __forceinline__ void keep_proposal(Prop o, const QueryInfo& qi, int64_t ext_signed,
                                              int32_t ext_len, const int32_t* fq, uint32_t nf,
                                              const LogfTable& logt, const ChainParams& p,
                                              DeviceStatus* st, uint32_t gidx, Prop* props,
                                              int& np, bool& overflow) {
  bool keep = overlap_test(o, qi.signed_id, ext_signed, qi.len, ext_len, p);
  if (keep) {
    const uint32_t lo = lower_bound_i32(fq, nf, o.cb);
    const uint32_t hi = lower_bound_i32(fq, nf, o.ce + 1);
    const int32_t norm = max(o.ce - o.cb, o.ee - o.eb) - static_cast<int32_t>(hi - lo);
    keep = norm > 0;
    if (keep) {
      float rate = fdiv(fmul(static_cast<float>(o.clen), p.sample_rate), static_cast<float>(norm));
      rate = rate < 1.0f ? rate : 1.0f;
      const float x = fdiv(1.0f, rate);
      if (!(x < 16777216.0f)) raise_status(st, kDevLogDomain, 0, static_cast<int64_t>(gidx));
      o.div = fdiv(flye_logf(x, logt), static_cast<float>(p.k));
    }
  }
  if (keep) {
    if (np == kMaxProposals) {
      raise_status(st, kDevProposalOverflow, 0, static_cast<int64_t>(gidx));
      overflow = true;
    } else {
      props[np++] = o;
    }
  }
}

// The group's proposals sorted by score descending in libstdc++ order, the
// primary ones kept under max_divergence, as rows in the pool.  One thread.
__device__ __forceinline__ void finish_group(const Prop* props, int np, const QueryInfo& qi,
                                             uint32_t query, uint32_t ext_di, int32_t ext_len,
                                             uint32_t gidx, const ChainParams& p,
                                             OverlapRow* __restrict__ pool, uint64_t pool_cap,
                                             uint32_t* __restrict__ pool_count,
                                             uint32_t* __restrict__ group_rows,
                                             DeviceStatus* st) {
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
  int keep[kMaxProposals];
  int nk = 0;
  for (int t = 0; t < nprim; ++t)
    if (props[prim[t]].div < p.max_divergence) keep[nk++] = prim[t];
  group_rows[gidx] = static_cast<uint32_t>(nk);
  if (nk == 0) return;
  const uint32_t base = atomicAdd(pool_count, static_cast<uint32_t>(nk));
  if (base + nk > pool_cap) {
    raise_status(st, kDevProposalOverflow, 1, static_cast<int64_t>(gidx));
    return;
  }
  for (int t = 0; t < nk; ++t) {
    const Prop& o = props[keep[t]];
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
    r.div = o.div;
    r.group = gidx;
    r.rank = static_cast<uint32_t>(t);
    pool[base + t] = r;
  }
}

}  // namespace cuflye
