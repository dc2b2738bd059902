// run_chain.cu — chaining of a target group over its runs.
//
// A group's hits in sort order (its axis: cur pos, or ext pos when ext_len >
// cur_len) are its pieces one after another; a piece's elements rise by one in
// cur and ext pos.  Flye's chaining over single hits
// (tools/replay_overlap_chains.py:280-346) follows from the pieces:
//
// DP.  An element inside a piece ends its scan at the element before it (jump
// divergence 0, closer than k), so its score is one more and its link i - 1.
// For a piece's first element, the elements of an earlier piece lie on one
// diagonal: going back, the score falls by one an element while the match grows
// by at most one and the gap cost stays, so only the last acceptable element
// of a piece (the last one before the scanning element in both positions) can
// beat the running maximum.  The scan therefore visits one candidate a piece.
//
// Equal axis positions.  Hits that share an axis position have an order only
// libstdc++'s sort knows.  Runs that overlap along the axis are cut wherever
// one of them starts or ends, so pieces that share a position share all of
// theirs (a tie cluster).  A scan's result depends on an order inside a cluster
// only if two or more of its candidates beat the running maximum and the
// greatest is not the only one of its score, or another one of them would end
// the scan.  An element inside a piece also meets the cluster's other elements
// one position back before its own predecessor; scores inside a cluster rise
// together, so one comparison of the first scores tells whether such a one could
// ever be its link.  Groups where the order could matter, and the ones the
// backtrack finds to depend on an order among equal scores, are left open: the
// hit path takes their hits.  Where the group repeats a cur position, the
// introsort of all its query's hits decides their order.
//
// Backtrack.  A walk clears a piece from some element down to its first, or to
// the part cleared before, so what is cleared of a piece is always a prefix,
// and the live element of the highest score is always the end of a piece.
#include <algorithm>
#include <climits>
#include <cstdint>

#include "common.cuh"
#include "kernels.h"
#include "proposals.cuh"
#include "runs.h"

namespace cuflye {
namespace {

constexpr int kWarpsPerBlock = 8;

__device__ __forceinline__ void list_group(const RunTables& t, uint32_t g, uint32_t npieces) {
  const int c = run_class(npieces);
  t.lists[c * t.max_groups + atomicAdd(t.counts + kRcList + c, 1u)] = g;
}

// Leaves a group to the hit path.
__device__ __forceinline__ void leave_open(const RunTables& t, uint32_t g) {
  t.open_list[atomicAdd(t.counts + kRcOpen, 1u)] = g;
}

// Group number li of the class lists (longest class first).
__device__ __forceinline__ uint32_t listed_group(const RunTables& t, uint32_t li) {
  int c = 0;
  for (; c + 1 < kRunClasses; ++c) {
    const uint32_t n = t.counts[kRcList + c];
    if (li < n) break;
    li -= n;
  }
  return t.lists[c * t.max_groups + li];
}

__device__ __forceinline__ uint32_t listed_total(const RunTables& t) {
  uint32_t n = 0;
#pragma unroll
  for (int c = 0; c < kRunClasses; ++c) n += t.counts[kRcList + c];
  return n;
}

__device__ __forceinline__ uint32_t next_item(uint32_t* counter) {
  uint32_t v = 0;
  if ((threadIdx.x & 31) == 0) v = atomicAdd(counter, 1u);
  return __shfl_sync(0xffffffffu, v, 0);
}

// ---------------------------------------------------------------- order

__device__ __forceinline__ void load_run(const RunTables& t, uint64_t i, bool es, int32_t& a,
                                         int32_t& b, int32_t& l) {
  const int32_t c = static_cast<int32_t>(t.keys[i] & 0xffffffffu);
  const int32_t e = static_cast<int32_t>(t.vals[i]);
  a = es ? e : c;
  b = es ? c : e;
  l = static_cast<int32_t>(t.rlen[i]);
}

// Piece slots of run j (in axis order) of a group without overlaps.
__device__ __forceinline__ void store_piece(const RunTables& t, uint64_t slot, int32_t a,
                                            int32_t b, int32_t l) {
  t.pa[slot] = a;
  t.pb[slot] = b;
  t.pl[slot] = l;
}

// Groups of up to 32 runs, a warp each: runs sorted in registers.  Groups
// whose runs overlap along the axis go to the block kernel.
__global__ void __launch_bounds__(kWarpsPerBlock * 32) order_small_kernel(RunTables t) {
  const int lane = threadIdx.x & 31;
  const uint32_t cnt = t.counts[kRcSort];
  const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
  for (uint32_t li = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); li < cnt; li += nwarps) {
    const uint32_t g = t.sort_lists[li];
    const RunGroup rg = t.groups[g];
    const uint32_t n = rg.nruns;
    const bool in = lane < static_cast<int>(n);
    int32_t a = 0, b = 0, l = 0;
    if (in) load_run(t, rg.run0 + lane, rg.flags & kRunExt, a, b, l);
    uint64_t key = in ? (static_cast<uint64_t>(static_cast<uint32_t>(a)) << 5) | lane : ~0ull;
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
      for (int st = size >> 1; st > 0; st >>= 1) {
        const uint64_t o = __shfl_xor_sync(0xffffffffu, key, st);
        const bool up = (lane & size) == 0, low = (lane & st) == 0;
        if ((o < key) == (up == low)) key = o;
      }
    }
    const int src = static_cast<int>(key & 31u);
    a = static_cast<int32_t>(key >> 5);
    b = __shfl_sync(0xffffffffu, b, src);
    l = __shfl_sync(0xffffffffu, l, src);
    int32_t inc = in ? a + l : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc = max(inc, y);
    }
    const int32_t before = __shfl_up_sync(0xffffffffu, inc, 1);
    if (__any_sync(0xffffffffu, in && lane > 0 && a < before)) {
      if (lane == 0)
        t.sort_lists[t.max_groups + atomicAdd(t.counts + kRcSort + 1, 1u)] = g;
      continue;
    }
    const uint64_t slot = rg.run0 + g;
    const int32_t l0 = __shfl_sync(0xffffffffu, l, 0);
    if (in) {
      if (lane == 0) {
        store_piece(t, slot, a, b, 1);
        const int32_t rest = l > 1 ? 1 : 0;
        store_piece(t, slot + 1, a + rest, b + rest, l - rest);
      } else {
        store_piece(t, slot + 1 + lane, a, b, l);
      }
    }
    if (lane == 0) {
      t.groups[g].piece0 = slot + (l0 > 1 ? 0u : 1u);
      t.groups[g].npieces = n + (l0 > 1 ? 1u : 0u);
      list_group(t, g, n + (l0 > 1 ? 1u : 0u));
    }
  }
}

template <int CAP, int PCAP>
struct OrderSmem {
  uint64_t rk[CAP];       // runs: axis << 32 | run
  int32_t ms[CAP];        // greatest end of the runs before
  uint32_t cuts[2 * CAP];  // where runs start and end, sorted
  uint64_t pk[PCAP];      // pieces: axis << 32 | slot in pb / pl
  int32_t pb[PCAP], pl[PCAP];
  int32_t wmax[32];
  uint32_t item, np, base;
  bool over, room;  // more pieces than pk holds; spare slots found
};

// np consecutive spare slots, or false when fewer are left.  A group that sees
// that it does not fit leaves the cursor where it is: smaller ones may still find
// room.  (One addition a claim: a compare-and-swap loop, which would also keep what
// a lost race for the last slots spends, waits a round trip for each claim of
// another block; all reads of a 1 Mb genome at 20x: 4.36 -> 4.70 ms.)
__device__ __forceinline__ bool claim_spares(const RunTables& t, uint32_t np, uint32_t& base) {
  if (*reinterpret_cast<volatile unsigned long long*>(t.spare_cursor) + np > t.spare_cap)
    return false;
  const unsigned long long at = atomicAdd(t.spare_cursor, static_cast<unsigned long long>(np));
  base = static_cast<uint32_t>(at);
  return at + np <= t.spare_cap;
}

// Bitonic sort of key[0, n) (room up to a power of two).
template <int BLOCK, class K>
__device__ void block_sort(K* key, uint32_t n) {
  uint32_t n2 = 1;
  while (n2 < n) n2 <<= 1;
  for (uint32_t i = n + threadIdx.x; i < n2; i += BLOCK) key[i] = ~static_cast<K>(0);
  __syncthreads();
  for (uint32_t size = 2; size <= n2; size <<= 1) {
    for (uint32_t st = size >> 1; st > 0; st >>= 1) {
      for (uint32_t i = threadIdx.x; i < n2 / 2; i += BLOCK) {
        const uint32_t lo = 2 * i - (i & (st - 1)), hi = lo + st;
        const K x = key[lo], y = key[hi];
        if ((x > y) == ((lo & size) == 0)) {
          key[lo] = y;
          key[hi] = x;
        }
      }
      __syncthreads();
    }
  }
}

// Pieces of the run [a, e) as act(axis pos, length): cut at every start and
// end of a run inside it, and after the group's first position a0.
template <class Act>
__device__ __forceinline__ void cut_run(const uint32_t* cuts, uint32_t ncuts, int32_t a,
                                        int32_t e, int32_t a0, Act act) {
  int32_t x = a;
  if (a == a0) {
    act(x, 1);
    ++x;
  }
  uint32_t lo = 0, hi = ncuts;  // first cut beyond x
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (static_cast<int32_t>(cuts[mid]) <= x)
      lo = mid + 1;
    else
      hi = mid;
  }
  while (x < e) {  // e is a cut
    const int32_t y = static_cast<int32_t>(cuts[lo]);
    act(x, y - x);
    x = y;
    while (lo < ncuts && static_cast<int32_t>(cuts[lo]) <= x) ++lo;
  }
}

// Groups of MIN < runs <= CAP, a block each, cut into up to PCAP pieces.  The
// last kernel also takes the groups that needed more pieces than the one
// before holds; what it cannot hold stays open.
template <int BLOCK, int MIN, int CAP, int PCAP, bool LAST>
__global__ void __launch_bounds__(BLOCK) order_block_kernel(RunTables t, uint32_t* work) {
  extern __shared__ __align__(16) unsigned char order_raw[];
  OrderSmem<CAP, PCAP>& sm = *reinterpret_cast<OrderSmem<CAP, PCAP>*>(order_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t cnt = t.counts[kRcSort + 1];
  for (;;) {
    __syncthreads();
    if (tid == 0) sm.item = atomicAdd(work, 1u);
    __syncthreads();
    const uint32_t li = sm.item;
    if (li >= cnt) break;
    const uint32_t g = t.sort_lists[t.max_groups + li];
    const RunGroup rg = t.groups[g];
    const uint32_t n = rg.nruns;
    if (LAST ? n <= MIN && !(rg.flags & kRunLarge) : n > CAP) continue;
    if (n > CAP) {
      if (tid == 0) leave_open(t, g);
      continue;
    }
    const bool es = rg.flags & kRunExt;
    for (uint32_t i = tid; i < n; i += BLOCK) {
      const uint32_t a = es ? t.vals[rg.run0 + i]
                            : static_cast<uint32_t>(t.keys[rg.run0 + i] & 0xffffffffu);
      sm.rk[i] = (static_cast<uint64_t>(a) << 32) | i;
    }
    __syncthreads();
    block_sort<BLOCK>(sm.rk, n);
    const uint32_t* rlen = t.rlen + rg.run0;
    // greatest end of the runs before each run: thread t owns a slice
    const uint32_t per = (n + BLOCK - 1) / BLOCK;
    const uint32_t i0 = min(n, tid * per), i1 = min(n, i0 + per);
    int32_t mx = 0;
    for (uint32_t i = i0; i < i1; ++i) {
      const int32_t a = static_cast<int32_t>(sm.rk[i] >> 32);
      const int32_t e = a + static_cast<int32_t>(rlen[sm.rk[i] & 0xffffffffu]);
      sm.cuts[2 * i] = static_cast<uint32_t>(a);
      sm.cuts[2 * i + 1] = static_cast<uint32_t>(e);
      sm.ms[i] = mx;
      mx = max(mx, e);
    }
    int32_t inc = mx;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc = max(inc, y);
    }
    if (lane == 31) sm.wmax[warp] = inc;
    __syncthreads();
    int32_t before = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) before = 0;
    for (int w = 0; w < warp; ++w) before = max(before, sm.wmax[w]);
    bool over = false;
    for (uint32_t i = i0; i < i1; ++i)
      over |= static_cast<int32_t>(sm.rk[i] >> 32) < max(sm.ms[i], before);
    if (tid == 0) {
      sm.np = 0;
      sm.over = false;
    }
    if (!__syncthreads_or(over)) {  // only out of order: one piece a run
      const uint64_t slot = rg.run0 + g;
      const uint32_t r0 = static_cast<uint32_t>(sm.rk[0] & 0xffffffffu);
      const uint32_t l0 = rlen[r0];
      for (uint32_t i = tid; i < n; i += BLOCK) {
        int32_t a, b, l;
        load_run(t, rg.run0 + (sm.rk[i] & 0xffffffffu), es, a, b, l);
        if (i == 0) {
          store_piece(t, slot, a, b, 1);
          const int32_t rest = l > 1 ? 1 : 0;
          store_piece(t, slot + 1, a + rest, b + rest, l - rest);
        } else {
          store_piece(t, slot + 1 + i, a, b, l);
        }
      }
      if (tid == 0) {
        t.groups[g].piece0 = slot + (l0 > 1 ? 0u : 1u);
        t.groups[g].npieces = n + (l0 > 1 ? 1u : 0u);
        list_group(t, g, n + (l0 > 1 ? 1u : 0u));
      }
      continue;
    }
    block_sort<BLOCK>(sm.cuts, 2 * n);
    const int32_t a0 = static_cast<int32_t>(sm.rk[0] >> 32);
    for (uint32_t i = tid; i < n; i += BLOCK) {
      int32_t a, b, l;
      load_run(t, rg.run0 + (sm.rk[i] & 0xffffffffu), es, a, b, l);
      uint32_t m = 0;
      cut_run(sm.cuts, 2 * n, a, a + l, a0, [&](int32_t, int32_t) { ++m; });
      uint32_t d = m <= PCAP ? atomicAdd(&sm.np, m) : PCAP;
      if (d + m > PCAP) {
        sm.over = true;
        continue;
      }
      cut_run(sm.cuts, 2 * n, a, a + l, a0, [&](int32_t x, int32_t len) {
        sm.pk[d] = (static_cast<uint64_t>(static_cast<uint32_t>(x)) << 32) | d;
        sm.pb[d] = b + (x - a);
        sm.pl[d] = len;
        ++d;
      });
    }
    __syncthreads();
    const uint32_t np = sm.np;
    if (sm.over && !LAST) {  // for the last kernel (over does not change until the next group)
      if (tid == 0) t.groups[g].flags = rg.flags | kRunLarge;
      continue;
    }
    if (tid == 0) sm.room = !sm.over && claim_spares(t, np, sm.base);
    __syncthreads();
    if (!sm.room) {
      if (tid == 0) leave_open(t, g);
      continue;
    }
    block_sort<BLOCK>(sm.pk, np);
    const uint64_t slot = t.spare0 + sm.base;
    for (uint32_t i = tid; i < np; i += BLOCK) {
      const uint32_t d = static_cast<uint32_t>(sm.pk[i] & 0xffffffffu);
      store_piece(t, slot + i, static_cast<int32_t>(sm.pk[i] >> 32), sm.pb[d], sm.pl[d]);
    }
    if (tid == 0) {
      t.groups[g].piece0 = slot;
      t.groups[g].npieces = np;
      t.groups[g].flags = (rg.flags & ~kRunLarge) | kRunTies;
      list_group(t, g, np);
    }
  }
}

// ---------------------------------------------------------------- DP

// The last element of a piece (a, b, l; first score s) that lies before (ai, bi)
// in both positions, as a predecessor: its score, offset, and whether an
// update by it ends the scan.
struct Candidate {
  int32_t score;  // INT_MIN: none
  int32_t off;
  bool ends;
};

__device__ __forceinline__ Candidate candidate(bool valid, int32_t ai, int32_t bi, int32_t a,
                                               int32_t b, int32_t l, int32_t s,
                                               const ChainParams& p) {
  const int32_t off = min(l, min(ai - a, bi - b)) - 1;
  const int32_t da = ai - a - off, db = bi - b - off;
  const int32_t jd = abs(da - db);
  const bool acc = valid && off >= 0 && da < p.max_jump && db < p.max_jump && jd <= p.max_gap;
  const float pen = jd > p.gap_jump_threshold ? p.large_gap_penalty : p.small_gap_penalty;
  const int32_t gc = __float2int_rz(__fmul_rn(pen, static_cast<float>(jd)));
  Candidate c;
  c.score = acc ? s + off + min(min(da, db), p.k) - gc : INT_MIN;
  c.off = off;
  c.ends = acc && jd == 0 && da < p.k;
  return c;
}

// One round of a scan over 32 candidates in scan order (lane 0 first), as
// Flye visits them: the first that beats the running maximum updates it, an
// update by one that ends the scan ends it.  ax: the candidates' axis
// positions (tie clusters: neighbours with the same one).  open: set when the
// order within a cluster could matter.
__device__ __forceinline__ void scan_round(const Candidate& c, int32_t ax, bool valid, bool ties,
                                           uint32_t j, int32_t& best, uint32_t& bestj,
                                           int32_t& bestoff, bool& ended, bool& open) {
  const int lane = threadIdx.x & 31;
  const bool acc = c.score != INT_MIN;
  if (!__any_sync(0xffffffffu, acc)) return;
  int32_t incl = c.score;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl = max(incl, o);
  }
  int32_t excl = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane == 0) excl = INT_MIN;
  const bool upd = acc && c.score > max(best, excl);
  const unsigned bm = __ballot_sync(0xffffffffu, upd && c.ends);
  const int bl = bm ? __ffs(bm) - 1 : 31;
  if (ties) {
    const int32_t pax = __shfl_up_sync(0xffffffffu, ax, 1);
    const bool pvalid = __shfl_up_sync(0xffffffffu, valid, 1);
    unsigned same = __ballot_sync(0xffffffffu, lane > 0 && valid && pvalid && ax == pax);
    while (same) {
      const int f = __ffs(same) - 2;  // the cluster's first lane
      const unsigned gaps = ~(same >> (f + 1));
      const int last = f + (gaps ? __ffs(gaps) - 1 : 31);
      same &= last >= 31 ? 0u : 0xffffffffu << (last + 1);
      if (f > bl) break;
      const int32_t from = max(best, __shfl_sync(0xffffffffu, excl, f));
      const bool above = acc && lane >= f && lane <= last && c.score > from;
      if (__popc(__ballot_sync(0xffffffffu, above)) >= 2) {
        const int32_t top = __reduce_max_sync(0xffffffffu, above ? c.score : INT_MIN);
        const int tops = __popc(__ballot_sync(0xffffffffu, above && c.score == top));
        if (tops > 1 || __any_sync(0xffffffffu, above && c.ends && c.score != top)) open = true;
      }
    }
  }
  const int32_t nb = max(best, __shfl_sync(0xffffffffu, incl, bl));
  if (nb > best) {
    const unsigned um = __ballot_sync(0xffffffffu, upd && lane <= bl && c.score == nb);
    const int w = __ffs(um) - 1;
    bestj = __shfl_sync(0xffffffffu, j, w);
    bestoff = __shfl_sync(0xffffffffu, c.off, w);
    best = nb;
  }
  ended = bm != 0;
}

// Inclusive scans over the warp.
__device__ __forceinline__ int32_t scan_add(int32_t x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}
__device__ __forceinline__ int32_t scan_max(int32_t x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x = max(x, y);
  }
  return x;
}

constexpr int32_t kNoScore = -(1 << 30);

// One warp a group, 32 pieces (a chunk) at a time.
//
// In a chain each piece links to the end of the one before it, and no other
// piece can do better: the piece before is visited first, and an older one
// scores its end plus k at most.  So the warp scores a stretch of pieces as if
// that were so with one prefix sum, checks it with one prefix maximum (the
// greatest end before each piece's predecessor), and keeps what comes before the
// first piece that fails.  That piece is scanned: against the 32 pieces before
// it, which the warp's registers hold (piece j in lane j mod 32), and against
// older ones only while the greatest end among them could still beat the best
// found.
//
// Bound by issue: a scan costs about 100 instructions a piece, a stretch
// about 4.
__global__ void __launch_bounds__(kWarpsPerBlock * 32) run_dp_kernel(RunTables t, ChainParams p,
                                                                     uint32_t* work) {
  const int lane = threadIdx.x & 31;
  const uint32_t cnt = listed_total(t);
  for (uint32_t li = next_item(work); li < cnt; li = next_item(work)) {
    const uint32_t gidx = listed_group(t, li);
    const RunGroup g = t.groups[gidx];
    const uint64_t base = g.piece0;
    const uint32_t n = g.npieces;
    const bool ties = g.flags & kRunTies;
    int32_t qa = 0, qb = 0, ql = 0, qs = 0;  // the chunk before: this lane's piece
    int32_t qmax = kNoScore;     // greatest end of that chunk's pieces before this lane's
    int32_t older = kNoScore;    // greatest end of the pieces before that chunk
    int32_t na = 0, nb = 0, nl = 0;  // the next chunk, loaded ahead
    int32_t s_prev = 0, e_prev = 0;  // score and end of the piece before the next one
    int32_t big = kNoScore;          // greatest end of the pieces before that one
    bool open = false;
    uint32_t first_tied = 0;  // pieces in a tie cluster at the first position
    bool ask_first = false;   // left open only for which of them is element 0
    if (lane < static_cast<int>(n)) {
      na = t.pa[base + lane];
      nb = t.pb[base + lane];
      nl = t.pl[base + lane];
    }
    for (uint32_t i0 = 0; i0 < n && !open; i0 += 32) {
      const int32_t ca = na, cb = nb, cl = nl;
      int32_t cs = 0;
      if (i0 + 32 + lane < n) {
        na = t.pa[base + i0 + 32 + lane];
        nb = t.pb[base + i0 + 32 + lane];
        nl = t.pl[base + i0 + 32 + lane];
      }
      const uint32_t len = min(32u, n - i0);
      uint32_t mk = kNoLink;
      int32_t mo = 0;
      // this piece after the end of the one before it: the score it would gain
      int32_t a1 = __shfl_up_sync(0xffffffffu, ca, 1), b1 = __shfl_up_sync(0xffffffffu, cb, 1),
              l1 = __shfl_up_sync(0xffffffffu, cl, 1);
      const int32_t la = __shfl_sync(0xffffffffu, qa, 31), lb = __shfl_sync(0xffffffffu, qb, 31),
                    ll = __shfl_sync(0xffffffffu, ql, 31);
      if (lane == 0) {
        a1 = la;
        b1 = lb;
        l1 = ll;
      }
      const Candidate pre = candidate(i0 + lane > 0, ca, cb, a1, b1, l1, 0, p);
      const int32_t gain = pre.score;
      bool ok = lane < static_cast<int>(len) && pre.score != INT_MIN && pre.off == l1 - 1;
      if (ties) {  // neither in a cluster nor after one
        int32_t a2 = __shfl_up_sync(0xffffffffu, a1, 1);
        const int32_t q30 = __shfl_sync(0xffffffffu, qa, 30);
        if (lane == 0) a2 = q30;
        ok = ok && ca != a1 && (a1 != a2 || i0 + lane < 2);
      }
      const unsigned okm = __ballot_sync(0xffffffffu, ok);
      uint32_t u = 0;
      if (i0 == 0) {
        // Element 0 of the group: score 0, no link.  In a tie cluster at the
        // group's first position any piece may be it, unless the group says
        // which; they score k, and if one of them becomes a link (with score 0
        // it never would) the group stays open for that
        const int32_t at0 = __shfl_sync(0xffffffffu, ca, 0);
        const bool at_first = lane < static_cast<int>(len) && ca == at0;
        first_tied = __popc(__ballot_sync(0xffffffffu, at_first));
        if (first_tied == 1) first_tied = 0;
        if (g.first) first_tied = 0;
        s_prev = first_tied || g.first > 1 ? p.k : 0;
        e_prev = s_prev;
        if (lane == 0) {
          cs = s_prev;
          if (ties) t.ps[base] = s_prev;
        }
        if (ties) __syncwarp();
        u = 1;
      }
      while (u < len && !open) {
        const unsigned stop = ~okm & (0xffffffffu << u);
        const uint32_t r = stop ? static_cast<uint32_t>(__ffs(stop) - 1) : 32u;
        if (r >= u + 3) {  // a stretch worth its scans
          const bool in = lane >= static_cast<int>(u) && lane < static_cast<int>(r);
          const int32_t s = s_prev + scan_add(in ? gain : 0);
          const int32_t e = s + cl - 1;
          const int32_t em = scan_max(in ? e : kNoScore);
          const int32_t em2 = __shfl_up_sync(0xffffffffu, em, 2);
          int32_t before = big;
          if (lane > static_cast<int>(u)) before = max(before, e_prev);
          if (lane > static_cast<int>(u) + 1) before = max(before, em2);
          const bool holds = in && s > p.k && (pre.ends || before + p.k <= s);
          const unsigned fail = ~__ballot_sync(0xffffffffu, holds) & (0xffffffffu << u);
          const uint32_t f = fail ? static_cast<uint32_t>(__ffs(fail) - 1) : 32u;
          if (f > u) {
            if (in && lane < static_cast<int>(f)) {
              cs = s;
              mk = i0 + lane - 1;
              mo = l1 - 1;
              if (ties) t.ps[base + i0 + lane] = s;
            }
            const int32_t ef1 = __shfl_sync(0xffffffffu, e, static_cast<int>(f - 1));
            const int32_t emf = __shfl_sync(0xffffffffu, em, static_cast<int>(max(f, 2u) - 2));
            big = max(big, e_prev);
            if (f >= u + 2) big = max(big, emf);
            e_prev = ef1;
            s_prev = __shfl_sync(0xffffffffu, s, static_cast<int>(f - 1));
            u = f;
            if (ties) __syncwarp();
            continue;
          }
        }
        // scan piece i0 + u
        const uint32_t i = i0 + u;
        const int32_t ai = __shfl_sync(0xffffffffu, ca, u);
        const int32_t bi = __shfl_sync(0xffffffffu, cb, u);
        const int32_t li_ = __shfl_sync(0xffffffffu, cl, u);
        const bool now = lane < static_cast<int>(u);  // the ring: this chunk's pieces so far
        const int32_t ra = now ? ca : qa, rb = now ? cb : qb, rl = now ? cl : ql,
                      rs = now ? cs : qs;
        const bool valid = now || i0 > 0;
        const Candidate c = candidate(valid, ai, bi, ra, rb, rl, rs, p);
        int32_t best = 0;
        uint32_t bestj = kNoLink;
        int32_t bestoff = 0;
        bool ended = false;
        // a tie cluster astride two rounds belongs to the later one: the
        // oldest pieces of this round that share the next one's position
        uint32_t held = 0;
        const uint32_t s0 = (i - 1) & 31;  // the lane of piece i - 1
        if (ties || __any_sync(0xffffffffu, c.ends)) {
          // in scan order: position d is the lane of piece i - 1 - d
          const int src = static_cast<int>((s0 - lane) & 31);
          Candidate o;
          o.score = __shfl_sync(0xffffffffu, c.score, src);
          o.off = __shfl_sync(0xffffffffu, c.off, src);
          o.ends = __shfl_sync(0xffffffffu, c.ends, src);
          const int32_t oax = __shfl_sync(0xffffffffu, ra, src);
          bool ov = lane < static_cast<int>(min(i, 32u));
          if (ties && i > 32) {
            const bool hold = oax == t.pa[base + i - 33];
            held = __popc(__ballot_sync(0xffffffffu, hold));
            if (hold) {
              ov = false;
              o.score = INT_MIN;
              o.ends = false;
            }
          }
          scan_round(o, oax, ov, ties, i - 1 - lane, best, bestj, bestoff, ended, open);
        } else {
          const int32_t m = __reduce_max_sync(0xffffffffu, c.score);
          if (m > 0) {
            const unsigned bal = __ballot_sync(0xffffffffu, c.score == m);
            // bit d of the rotated word: the lane of piece i - 1 - d
            const unsigned rev = __brev(bal);
            const uint32_t d = __ffs(__funnelshift_r(rev, rev, 31 - s0)) - 1;
            best = m;
            bestj = i - 1 - d;
            bestoff = __shfl_sync(0xffffffffu, c.off, static_cast<int>((s0 - d) & 31));
          }
        }
        if (i > 32 && !ended) {
          const int32_t past = max(older, __shfl_sync(0xffffffffu, qmax, static_cast<int>(u)));
          if (held || past + p.k > best) {
            // beyond the jump along the axis from some piece on?  (held pieces
            // are the oldest: lane order d >= 32 - held)
            const uint32_t d = (s0 - lane) & 31;
            bool more = !__any_sync(0xffffffffu, d < 32 - held && ai - ra > p.max_jump);
            if (held == 32) {
              open = true;
              more = false;
            }
            for (int32_t c0 = static_cast<int32_t>(i + held) - 33; more && c0 >= 0;) {
              const int32_t jj = c0 - lane;
              bool v = jj >= 0;
              int32_t a = 0, b = 0, l = 0, s = 0;
              if (v) {
                a = t.pa[base + jj];
                b = t.pb[base + jj];
                l = t.pl[base + jj];
                s = __ldcg(t.ps + base + jj);
              }
              held = 0;
              if (ties && c0 >= 32) {
                const bool hold = a == t.pa[base + c0 - 32];
                held = __popc(__ballot_sync(0xffffffffu, hold));
                if (hold) v = false;
                if (held == 32) open = true;
              }
              const Candidate x = candidate(v, ai, bi, a, b, l, s, p);
              scan_round(x, a, v, ties, static_cast<uint32_t>(jj), best, bestj, bestoff, ended,
                         open);
              if (ended || open || __any_sync(0xffffffffu, v && ai - a > p.max_jump) ||
                  (held == 0 && past + p.k <= best))
                break;
              c0 -= 32 - static_cast<int32_t>(held);
            }
          }
        }
        const int32_t si = i + 1 == g.first ? 0 : max(best, p.k);
        if (ties) {
          if (best > p.k && bestj < first_tied) ask_first = open = true;
          // the cluster so far: could the elements inside one of two pieces
          // link into the other (one axis position back, so on a lower second
          // position)?
          const bool mate = valid && ra == ai;
          const int32_t d = bi - rb, jd = abs(d);
          const float pen = jd > p.gap_jump_threshold ? p.large_gap_penalty : p.small_gap_penalty;
          const int32_t gc = __float2int_rz(__fmul_rn(pen, static_cast<float>(jd)));
          const bool close = jd <= p.max_gap && jd + 1 < p.max_jump;
          const bool unsafe = mate && li_ > 1 && close && !(d > 0 ? si > rs - gc : rs > si - gc);
          const unsigned mates = __ballot_sync(0xffffffffu, mate);
          if (__any_sync(0xffffffffu, unsafe) || mates == 0xffffffffu) {
            open = true;
            ask_first = false;
          }
        }
        if (lane == static_cast<int>(u)) {
          cs = si;
          mk = best > p.k ? bestj : kNoLink;
          mo = best > p.k ? bestoff : 0;
          if (ties) t.ps[base + i] = si;  // a held piece is read back before the chunk's store
        }
        if (ties) __syncwarp();
        big = max(big, e_prev);
        s_prev = si;
        e_prev = si + li_ - 1;
        ++u;
      }
      if (lane < static_cast<int>(len)) {
        t.ps[base + i0 + lane] = cs;
        t.pk[base + i0 + lane] = mk;
        t.po[base + i0 + lane] = mo;
      }
      __syncwarp();
      older = max(older, __reduce_max_sync(0xffffffffu, i0 > 0 ? qs + ql - 1 : kNoScore));
      qa = ca;
      qb = cb;
      ql = cl;
      qs = cs;
      const int32_t em = scan_max(cs + cl - 1);
      qmax = __shfl_up_sync(0xffffffffu, em, 1);
      if (lane == 0) qmax = kNoScore;
    }
    if (open && lane == 0) {
      t.groups[gidx].flags = g.flags | kRunOpen | (ask_first ? kRunFirst : 0u);
      leave_open(t, gidx);
    }
  }
}

// ---------------------------------------------------------------- backtrack

// Pieces a group may have for its walk tables to lie in shared memory.
constexpr uint32_t kWalkCap = 256;

struct WalkSmem {
  uint32_t link[kWalkCap];
  int32_t off[kWalkCap];
  int32_t done[kWalkCap];
  int32_t upto[kWalkCap];
  int32_t end[kWalkCap];
};

struct WalkTables {
  const uint32_t* link;  // per piece: the piece its first element links to (kNoLink: none) ...
  const int32_t* off;    // ... and the element of it
  int32_t* done;         // elements cleared, from the first on
  int32_t* upto;         // elements of the pieces up to this one
  int32_t* end;          // score of the last element, kNoScore if it has no link
  uint32_t* marks;       // per piece: the last tie round that walked it, and
                         // what was cleared of it before that round
  __device__ __forceinline__ int32_t before(uint32_t i) const { return i ? upto[i - 1] : 0; }
  __device__ __forceinline__ int32_t len(uint32_t i) const { return upto[i] - before(i); }
};

// Notes that a tie round walks piece r, d of whose elements are cleared.
__device__ __forceinline__ void mark_walked(const WalkTables& w, uint32_t r, uint32_t round,
                                            int32_t d) {
  uint32_t* m = w.marks + 2ull * r;
  if (m[0] != round) m[1] = static_cast<uint32_t>(d);
  m[0] = round;
}

// Walk from element off of piece r: first element, chain length as Flye's walk
// counts them; what it visits becomes cleared.  round > 0: `met` tells whether
// the walk ended on a linked element that another walk of the round cleared (an
// element cleared before the round ends every walk that reaches it, as one
// without a link does).  Pieces that link to the end of the piece before
// and are not yet cleared are passed 32 at a time.
__device__ __forceinline__ void walk_pieces(const WalkTables& w, uint32_t r, int32_t off,
                                            uint32_t round, uint32_t& fr, int32_t& fo,
                                            int32_t& clen, bool& met) {
  const int lane = threadIdx.x & 31;
  clen = 0;
  for (;;) {
    const int32_t j = static_cast<int32_t>(r) - lane;
    bool pass = false;
    int32_t l = 0;
    if (j > 0) {
      l = w.len(j);
      pass = w.link[j] == static_cast<uint32_t>(j - 1) && w.off[j] == w.len(j - 1) - 1 &&
             w.done[j] == 0;
    }
    const unsigned held = ~__ballot_sync(0xffffffffu, pass);
    const int np = held ? __ffs(held) - 1 : 32;  // pieces passed
    if (np > 0) {
      if (lane < np) {
        const int32_t top = lane == 0 ? off : l - 1;
        w.done[j] = top + 1;
        if (round) mark_walked(w, static_cast<uint32_t>(j), round, 0);
      }
      clen += off + 1 + w.before(r) - w.before(r - np + 1);
      __syncwarp();
      r -= np;
      off = w.len(r) - 1;
      if (np == 32) continue;
    }
    // piece r: down to z, and there stop if z is cleared or has no link
    const int32_t d = w.done[r];
    const uint32_t link = w.link[r];
    const int32_t z = off < d ? off : d > 0 ? d - 1 : 0;
    const bool linked = z > 0 || link != kNoLink;
    const bool stop = d > 0 || !linked;
    clen += off - z + 1;
    if (round && stop) {
      const uint32_t* m = w.marks + 2ull * r;
      met = linked && z < d && m[0] == round && z >= static_cast<int32_t>(m[1]);
    }
    __syncwarp();
    if (lane == 0) {
      if (off >= d) w.done[r] = off + 1;
      if (round) mark_walked(w, r, round, d);
    }
    __syncwarp();
    if (stop) {
      fr = r;
      fo = z;
      return;
    }
    off = w.off[r];
    r = link;
  }
}

// One warp a group.  Bound by the latency of each group's chain (tables loaded,
// walks, the searches of a proposal), so everything a walk reads is staged in
// shared memory, and the searches probe 32 places a round.
__global__ void __launch_bounds__(kWarpsPerBlock * 32, 4) run_backtrack_kernel(
    RunTables t, ChainParams p, const uint64_t* __restrict__ f_off,
    const int32_t* __restrict__ fpos, LogfTable logt, OverlapRow* __restrict__ pool,
    uint64_t pool_cap, uint32_t* __restrict__ group_rows, DeviceStatus* st, uint32_t* work) {
  __shared__ WalkSmem smem[kWarpsPerBlock];
  const int lane = threadIdx.x & 31;
  WalkSmem& sw = smem[threadIdx.x >> 5];
  const uint32_t cnt = listed_total(t);
  for (uint32_t li = next_item(work); li < cnt; li = next_item(work)) {
    const uint32_t gidx = listed_group(t, li);
    const RunGroup g = t.groups[gidx];
    if (g.flags & kRunOpen) continue;
    const uint64_t base = g.piece0;
    const uint32_t n = g.npieces;
    const bool es = g.flags & kRunExt;
    const QueryInfo qi = t.qinfo[g.query];
    const int64_t ext_signed = (g.ext_di & 1u) ? -t.idx.slot_signed[g.ext_di >> 1]
                                               : t.idx.slot_signed[g.ext_di >> 1];
    const int32_t* fq = fpos + f_off[g.query];
    const uint32_t nf = static_cast<uint32_t>(f_off[g.query + 1] - f_off[g.query]);
    const bool small = n <= kWalkCap;
    WalkTables w{sw.link, sw.off, sw.done, sw.upto, sw.end, t.pm + 2 * base};
    if (!small) {
      w.link = t.pk + base;
      w.off = t.po + base;
      w.done = t.pd + base;
      w.upto = t.pp + base;
      w.end = t.pe + base;
    }
    int32_t total = 0;
    for (uint32_t i0 = 0; i0 < n; i0 += 32) {
      const uint32_t i = i0 + lane;
      const bool in = i < n;
      const int32_t l = in ? t.pl[base + i] : 0;
      const int32_t upto = scan_add(l);
      if (in) {
        const uint32_t link = t.pk[base + i];
        if (small) {
          sw.link[i] = link;
          sw.off[i] = t.po[base + i];
        }
        w.done[i] = 0;
        w.upto[i] = total + upto;
        w.end[i] = l >= 2 || link != kNoLink ? t.ps[base + i] + l - 1 : kNoScore;
      }
      total += __shfl_sync(0xffffffffu, upto, 31);
    }
    __syncwarp();
    Prop props[kMaxProposals];
    int np = 0;
    bool overflow = false, ambiguous = false, multi = false;
    uint32_t round = 0;
    auto propose = [&](uint32_t r, uint32_t fr, int32_t fo, int32_t clen) {
      if (overflow) return;
      const int32_t l1 = w.len(r) - 1;
      const int32_t a0 = t.pa[base + fr] + fo, b0 = t.pb[base + fr] + fo;
      const int32_t a1 = t.pa[base + r] + l1, b1 = t.pb[base + r] + l1;
      Prop o;
      o.cb = es ? b0 : a0;
      o.ce = (es ? b1 : a1) + p.k - 1;
      o.eb = es ? a0 : b0;
      o.ee = (es ? a1 : b1) + p.k - 1;
      o.score = w.end[r] - (t.ps[base + fr] + fo) + p.k - 1;
      o.clen = clen;
      keep_proposal(o, qi, ext_signed, g.ext_len, fq, nf, p, st, gidx, props, np, overflow);
    };
    // Starts by score: the live linked element of the highest score next, always
    // the end of a piece.  Ends sharing the top score are walked in order; see
    // backtrack_kernel (chain.cu) for when Flye's order among them matters.
    for (;;) {
      int32_t bs = INT_MIN;
      uint32_t bi = kNoLink, bc = 0;
      for (uint32_t i = lane; i < n; i += 32) {
        const int32_t s = w.end[i];
        if (s == kNoScore || w.done[i] >= w.len(i)) continue;
        if (s > bs) {
          bs = s;
          bi = i;
          bc = 1;
        } else if (s == bs) {
          ++bc;
        }
      }
      const int32_t ms = __reduce_max_sync(0xffffffffu, bs);
      const uint32_t mc = __reduce_add_sync(0xffffffffu, bs == ms ? bc : 0u);
      if (mc == 0) break;
      const uint32_t mi = __reduce_min_sync(0xffffffffu, bs == ms ? bi : kNoLink);
      uint32_t fr = 0;
      int32_t fo = 0, clen = 0;
      bool met = false;
      if (mc == 1) {
        walk_pieces(w, mi, w.len(mi) - 1, 0, fr, fo, clen, met);
        propose(mi, fr, fo, clen);
        __syncwarp();
        continue;
      }
      // a tie round over the mc live ends of score ms
      if (round == 0) {
        for (uint32_t i = lane; i < n; i += 32) w.marks[2ull * i] = 0;
        __syncwarp();
      }
      ++round;
      const int np0 = np;
      bool clash = false;
      uint32_t left = mc;
      for (uint32_t i0 = mi & ~31u; i0 < n && left > 0 && !clash; i0 += 32) {
        const uint32_t i = i0 + lane;
        bool tied = false;
        if (i < n) tied = w.end[i] == ms && w.done[i] < w.len(i);
        unsigned tm = __ballot_sync(0xffffffffu, tied);
        while (tm && !clash) {
          const uint32_t r = i0 + __ffs(tm) - 1;
          tm &= tm - 1;
          --left;
          const int32_t l = w.len(r);
          if (w.done[r] >= l) {  // cleared by an earlier walk of this round
            clash = true;
            break;
          }
          met = false;
          walk_pieces(w, r, l - 1, round, fr, fo, clen, met);
          if (met) {
            clash = true;
            break;
          }
          propose(r, fr, fo, clen);
          __syncwarp();
        }
      }
      if (left > 0) clash = true;  // a tied end cleared before it was reached
      if (lane == 0 && !clash) {
        for (int i = np0; i < np && !clash; ++i)
          for (int j = i + 1; j < np; ++j)
            if (props[i].score == props[j].score) clash = true;
        if (np - np0 >= 2) multi = true;
      }
      clash = __shfl_sync(0xffffffffu, clash, 0);
      if (clash) {
        ambiguous = true;
        break;
      }
    }
    if (multi && np > 16) ambiguous = true;
    __syncwarp();
    if (lane != 0) continue;
    if (ambiguous) {
      t.groups[gidx].flags = g.flags | kRunOpen;
      leave_open(t, gidx);
    } else if (overflow) {
      group_rows[gidx] = 0;
    } else {
      finish_group(props, np, qi, g.query, g.ext_di, g.ext_len, gidx, logt, p, pool, pool_cap,
                   t.counts + kRcPool, group_rows, st);
    }
  }
}

}  // namespace

cudaError_t runs_order(const RunTables& t, int num_sms, cudaStream_t s) {
  if (t.max_groups == 0) return cudaSuccess;
  const uint64_t warps = (t.max_groups + kWarpsPerBlock - 1) / kWarpsPerBlock;
  count_launch();
  order_small_kernel<<<static_cast<unsigned>(std::min<uint64_t>(warps, 32ull * num_sms)),
                       kWarpsPerBlock * 32, 0, s>>>(t);
  auto mid = order_block_kernel<128, 0, 512, 2048, false>;
  auto big = order_block_kernel<512, 512, 4096, 8192, true>;
  cudaError_t e = cudaFuncSetAttribute(mid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(sizeof(OrderSmem<512, 2048>)));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(big, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(sizeof(OrderSmem<4096, 8192>)));
  if (e != cudaSuccess) return e;
  count_launch();
  mid<<<static_cast<unsigned>(std::min<uint64_t>(t.max_groups, 8ull * num_sms)), 128,
        sizeof(OrderSmem<512, 2048>), s>>>(t, t.counts + kRcWork + 1);
  count_launch();
  big<<<static_cast<unsigned>(std::min<uint64_t>(t.max_groups, num_sms)), 512,
        sizeof(OrderSmem<4096, 8192>), s>>>(t, t.counts + kRcWork + 2);
  return cudaGetLastError();
}

cudaError_t runs_dp(const RunTables& t, const ChainParams& p, int num_sms, int per_sm,
                    cudaStream_t s) {
  if (t.max_groups == 0) return cudaSuccess;
  int most = 0;
  cudaError_t e =
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&most, run_dp_kernel, kWarpsPerBlock * 32, 0);
  if (e != cudaSuccess) return e;
  most = std::max(most, 1);
  // warps take groups from a counter: the grid changes no result
  const uint64_t blocks = static_cast<uint64_t>(num_sms) * (per_sm > 0 ? std::min(per_sm, most) : most);
  const uint64_t need = (t.max_groups + kWarpsPerBlock - 1) / kWarpsPerBlock;
  count_launch();
  run_dp_kernel<<<static_cast<unsigned>(std::min(blocks, need)), kWarpsPerBlock * 32, 0, s>>>(
      t, p, t.counts + kRcWork + 3);
  return cudaGetLastError();
}

cudaError_t runs_backtrack(const RunTables& t, const ChainParams& p, const uint64_t* f_off,
                           const int32_t* fpos, const LogfTable& logt, OverlapRow* pool,
                           uint64_t pool_cap, uint32_t* group_rows, DeviceStatus* st, int num_sms,
                           int per_sm, cudaStream_t s) {
  if (t.max_groups == 0) return cudaSuccess;
  const uint64_t blocks = static_cast<uint64_t>(num_sms) * (per_sm > 0 ? std::min(per_sm, 4) : 4);
  const uint64_t need = (t.max_groups + kWarpsPerBlock - 1) / kWarpsPerBlock;
  count_launch();
  run_backtrack_kernel<<<static_cast<unsigned>(std::min(blocks, need)), kWarpsPerBlock * 32, 0,
                         s>>>(t, p, f_off, fpos, logt, pool, pool_cap, group_rows, st,
                              t.counts + kRcWork + 4);
  return cudaGetLastError();
}

}  // namespace cuflye
