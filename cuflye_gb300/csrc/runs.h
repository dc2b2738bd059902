// runs.h — launchers of the run path (runs.cu, run_chain.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.h"

namespace cuflye {

// A run: hits of one (query, ext id) pair at consecutive cur and ext
// positions, as long as it gets.  Runs are found and sorted like hits (key =
// (ext id << 32) | first cur pos, val = first ext pos).
//
// A piece: a run, or a part of one, of a group's chaining order.  Pieces of a
// group follow one another in its sort axis (cur pos, or ext pos when
// ext_len > cur_len), except pieces that share all of their axis positions (a
// tie cluster).  Element 0 of a group is a piece of its own.

enum : uint32_t {
  kRunExt = 1,      // sort axis: ext pos
  kRunCurTies = 2,  // two hits of the group share a cur pos
  kRunTies = 4,     // its pieces hold tie clusters
  kRunLarge = 16,   // more pieces than the smaller ordering kernel holds
  kRunOpen = 8,     // left to the hit path: its result may depend on an order of equal keys
  kRunFirst = 32,   // left open only for which piece of its first position is element 0
};

struct RunGroup {
  uint64_t piece0;  // first piece
  uint64_t run0;    // first run (KmerMatch order)
  uint32_t nruns, npieces;
  uint32_t nhits;
  uint32_t query, ext_di;
  int32_t ext_len;
  uint32_t flags;
  // 1 + the piece that is element 0, of several at the group's first position
  // (0: not known): found from the order of its hits, see runs_settle_first
  uint32_t first;
};

// Length classes of the surviving groups, longest first; list c holds the
// groups of class c at lists[c * cap ..].
constexpr int kRunClasses = 5;
#ifdef __CUDACC__
__device__ __forceinline__ int run_class(uint32_t npieces) {
  return npieces > 1024 ? 0 : npieces > 256 ? 1 : npieces > 64 ? 2 : npieces > 16 ? 3 : 4;
}
#endif

// Device counters of a pass (u32 words, zeroed by the caller).
enum : int {
  kRcList = 0,                        // kRunClasses: surviving groups by class
  kRcSort = kRunClasses,              // 2: groups whose runs need sorting (small, large)
  kRcOpen = kRcSort + 2,              // groups left to the hit path
  kRcExt = kRcOpen + 1,               // surviving ext-axis groups
  kRcPool = kRcExt + 1,               // rows in the pool
  kRcWork = kRcPool + 1,              // 5: work counters
  kRcWords = kRcWork + 6,             // one more, for an even number
};

struct RunTables {
  DeviceIndex idx;
  QueryBatch qb;
  const QueryInfo* qinfo = nullptr;
  const uint32_t* cbits = nullptr;  // per 32 windows: bit w = window is solid
  const uint64_t* keys = nullptr;   // sorted runs
  const uint32_t* vals = nullptr;
  uint64_t nruns = 0;
  const GroupInfo* bounds = nullptr;  // start, query and ext id of each group
  const uint64_t* ngroups = nullptr;  // on the device
  uint64_t max_groups = 0;
  uint32_t* rlen = nullptr;           // run lengths (hits)
  RunGroup* groups = nullptr;
  // pieces: nruns + max_groups slots for groups whose runs are pieces
  // (group g's runs from slot run0 + g), then spare slots for split groups
  int32_t *pa = nullptr, *pb = nullptr, *pl = nullptr;
  uint64_t spare0 = 0, spare_cap = 0;
  unsigned long long* spare_cursor = nullptr;
  int32_t* ps = nullptr;   // score of the piece's first element
  uint32_t* pk = nullptr;  // its link: piece of the group (kNoLink: none) ...
  int32_t* po = nullptr;   // ... and offset in it
  // the backtrack's tables of groups beyond shared memory: elements cleared,
  // elements up to each piece, end scores
  int32_t *pd = nullptr, *pp = nullptr, *pe = nullptr;
  uint32_t* pm = nullptr;  // tie-round marks, 2 words a piece
  uint32_t* lists = nullptr;       // kRunClasses * max_groups
  uint32_t* sort_lists = nullptr;  // 2 * max_groups
  uint32_t* open_list = nullptr;   // max_groups
  uint32_t* counts = nullptr;      // kRcWords
};
constexpr uint32_t kNoLink = 0xffffffffu;

// Neighbour bases of every stored entry: low nibble the base before the
// k-mer on the stored strand, high nibble the base after it (4: the target
// ends there).  nbr must hold 16 bytes past the last entry.
cudaError_t index_neighbours(const uint64_t* pos, uint64_t npos, const uint64_t* words,
                             const uint64_t* base_off, const int32_t* slot_len, int k,
                             uint8_t* nbr, cudaStream_t s);

// Per window its run starts (nstart), and a record (recs) for runs_emit where
// it has some or is filtered; per 32 windows the run starts, and the bits of
// solid and of filtered windows.
cudaError_t runs_count(const DeviceIndex& idx, const QueryBatch& q, uint4* recs, uint32_t* nstart,
                       uint32_t* cbits, uint32_t* fbits, uint32_t* tile_filt,
                       uint32_t* tile_start, int num_sms, cudaStream_t s);
// Each query's first run and first filtered position (nq + 1 entries each);
// totals (zeroed by the caller): [0] the most runs of a query, [1] and [2] all
// runs and filtered positions, [3] the queries in list (nq words): those of
// more than kRunSortCap and up to kRunSortLarge runs.
cudaError_t runs_query_offsets(const QueryBatch& q, const uint32_t* nstart,
                               const uint64_t* tile_off, const uint32_t* fbits,
                               const uint64_t* ftile_off, uint64_t* q_off, uint64_t* f_off,
                               unsigned long long* totals, uint32_t* list,
                               cudaStream_t s);
// The run starts in window order, then bucket order, and the filtered positions.
cudaError_t runs_emit(const DeviceIndex& idx, const QueryBatch& q, const uint4* recs,
                      const uint32_t* nstart, const uint64_t* tile_off, const uint32_t* fbits,
                      const uint64_t* ftile_off, uint64_t* keys, uint32_t* vals, int32_t* fpos,
                      cudaStream_t s);

// The runs of every query of up to on_chip (kRunSortCap or kRunSortLarge) runs
// sorted by ext id, in place and stable (longer ones come sorted, by match_radix),
// and the groups of each query.  longest, list, list_count: from runs_query_offsets.  work: two
// counters, zeroed by the caller.
constexpr uint32_t kRunSortCap = 4096, kRunSortLarge = 16384;
cudaError_t runs_sort(const uint64_t* q_off, uint32_t nq, uint64_t longest, uint32_t on_chip,
                      const uint32_t* list,
                      const unsigned long long* list_count, uint64_t* keys, uint32_t* vals,
                      int id_bits, uint32_t* q_groups, uint32_t* work, int num_sms,
                      cudaStream_t s);
// Start, query and ext id of each group; q_group: the scan of q_groups.
cudaError_t runs_bounds(const uint64_t* q_off, uint32_t nq, const uint64_t* keys,
                        const uint64_t* q_group, GroupInfo* bounds, int num_sms, cudaStream_t s);
// Run lengths, group prefilter, and the pieces of groups whose runs are in
// order already; the other survivors are listed for runs_order.
cudaError_t runs_groups(const RunTables& t, const ChainParams& p, int num_sms, cudaStream_t s);
// Sorts the listed groups' runs along their axis and splits runs that overlap.
cudaError_t runs_order(const RunTables& t, int num_sms, cudaStream_t s);
cudaError_t runs_dp(const RunTables& t, const ChainParams& p, int num_sms, int per_sm,
                    cudaStream_t s);
cudaError_t runs_backtrack(const RunTables& t, const ChainParams& p, const uint64_t* f_off,
                           const int32_t* fpos, const LogfTable& logt, OverlapRow* pool,
                           uint64_t pool_cap, uint32_t* group_rows, DeviceStatus* st, int num_sms,
                           int per_sm, cudaStream_t s);

// Open groups take the hit path's chaining, in batches: their hits in
// KmerMatch order (runs_expand), and the rows back into the pool.
struct OpenInfo {
  uint32_t group, query, nhits, flags;
};
struct OpenBatch {
  uint32_t n = 0;
  const uint32_t* list = nullptr;   // run groups
  const uint64_t* off = nullptr;    // first hit of each in the batch's arrays
  const uint32_t* src_q = nullptr;  // groups that repeat a cur position: their
                                    // query among the sorted ones, else kNoLink
  // hits of those queries in KmerMatch order (for the listed tie keys)
  const uint64_t* sorted_off = nullptr;
  const uint64_t* sorted_keys = nullptr;
  const uint32_t* sorted_vals = nullptr;
};
cudaError_t runs_open_info(const RunTables& t, uint32_t nopen, OpenInfo* out, cudaStream_t s);
// KmerMatch keys that two hits of such a group share, as (src_q, key), in
// any order and possibly repeated; *count counts them all, cap are stored.
cudaError_t runs_tie_keys(const RunTables& t, const OpenBatch& o, uint64_t* tie_q,
                          uint64_t* tie_key, unsigned long long* count, uint64_t cap,
                          cudaStream_t s);
// Hits and a GroupInfo per group; counts[0] / [1]: ext_list and dp_list.
cudaError_t runs_expand(const RunTables& t, const OpenBatch& o, uint64_t* keys, uint32_t* vals,
                        GroupInfo* groups, uint32_t* ext_list, uint32_t* dp_list,
                        uint32_t* counts, int num_sms, cudaStream_t s);
cudaError_t runs_append_rows(const OverlapRow* from, const uint32_t* nfrom, const uint32_t* list,
                             OverlapRow* pool, uint64_t pool_cap, uint32_t* pool_count,
                             DeviceStatus* st, int num_sms, cudaStream_t s);
// Open groups whose flags hold kRunFirst, once their hits are in Flye's order
// (keys, vals, groups: a batch's hits as chain_groups sorts them): their element
// 0 is set, their flags are cleared, and they are listed for runs_dp and
// runs_backtrack in lists / counts of a RunTables of their own.
cudaError_t runs_settle_first(const RunTables& t, const OpenBatch& o, const uint64_t* keys,
                              const uint32_t* vals, const GroupInfo* groups, uint32_t* lists,
                              uint32_t* counts, cudaStream_t s);
// The batch's groups that are still the hit path's (not settled) into dp_list,
// their number into *count (zeroed by the caller).
cudaError_t runs_unsettled(const RunTables& t, const OpenBatch& o, uint32_t* dp_list,
                           uint32_t* count, cudaStream_t s);
// group_rows[open_list[i]] = rows[i], for the groups that are not settled.
cudaError_t runs_fold_rows(const RunTables& t, const uint32_t* open_list, uint32_t nopen,
                           const uint32_t* rows, uint32_t* group_rows, cudaStream_t s);
// Pool rows to their places.
cudaError_t runs_scatter_rows(const OverlapRow* pool, const uint32_t* npool, uint64_t max_pool,
                              const uint32_t* kept, const uint64_t* kept_off, OverlapRow* rows,
                              cudaStream_t s);

}  // namespace cuflye
