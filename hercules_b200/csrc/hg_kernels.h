// hg_kernels.h -- launchers of the sm_100a kernels (host side declarations).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace hg {

// Raises one kernel's dynamic shared-memory limit on the current device
// before its first launch there.  cudaFuncSetAttribute acts on the current
// device only, so the "done" state is one bit per device (devices 0..63;
// higher ones set the attribute on every launch).  Two host threads making
// their first call at once may both set it, which is harmless: the value is
// the same.  One instance per (kernel, limit) call site, as a function-local
// static.
class SmemLimit {
 public:
  cudaError_t ensure(const void* func, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
    if (bit && (done_.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && bit) done_.fetch_or(bit, std::memory_order_acq_rel);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

constexpr int kEdWarps = 8;  // warps per block of the distance stream (32 where the staged query is large)
constexpr int kEdBlocksPerSm = 4;  // resident blocks per SM of the distance stream
constexpr int kWarpListCap = 256;  // per-warp candidate buffer (k <= kWarpListCap - 32)
constexpr int kMaxK = kWarpListCap - 32;
constexpr int kMaxLeavesSort = 8192;  // leaves whose sort / grouping arrays fit in shared memory
constexpr int kMergeCap = 8192;       // single-CTA bitonic merge capacity

// A routing node of the EAPCA tree: an internal node's split policy
// (hercules_node_split.h:21-34) and its children; a child < 0 is the leaf ~child.
struct DNode {
  int left, right;
  float value;
  short from, to;
  int idx;
  int pad;
};

struct Tree {
  const DNode* nodes;
  int root;  // >= 0 internal node, < 0 the leaf ~root
};

// The kernels of the plain path serve a group of queries per launch: grid.x is
// the query's slot in the group, and every per-query array below holds one
// entry (or one run of the stated stride) per slot.  Slots vary fastest, so
// the blocks of all queries of a group run side by side.

// Routing, LB_EAPCA of every leaf and the LB_SAX term table.
struct PrepArgs {
  const float* q;        // [slot][L]
  int L;
  Tree tree;
  int nleaves;
  const int* seg_off;    // leaf envelopes (CSR)
  const short* points;
  const float* sk;
  const float* bp;
  float* lb;             // [slot][nleaves]; NULL: no lower bounds
  float* sax_tab;        // [slot][16 x 256] LB_SAX terms; NULL: none
  int* approx_leaf;      // [slot]; NULL: no routing, and the state below is left alone
  uint32_t* bound;       // [slot] reset to +inf
  uint32_t* kslots;      // [slot][kMaxK] reset to +inf
  int* topk_count;       // [slot] reset to 0
  uint32_t* counters;    // [slot][8] reset to 0
};

// Stage 1 of the leaf scan: candidate leaves -> their rows, with LB_SAX its survivors
// (launch_lbsax_filter) or all of them (launch_list_rows).
struct FilterArgs {
  const uint8_t* sax;
  int L;
  int nleaves;
  const uint64_t* leaf_start;
  const uint32_t* leaf_size;
  const int* cand;              // [slot][nleaves + 1]
  const float* cand_lb;         // [slot][nleaves + 1] ascending
  const int* cand_count;        // [slot]
  const uint32_t* unit_prefix;  // [slot][nleaves + 2] exclusive prefix of 32-row units per candidate
  const uint32_t* row_prefix;   // [slot][nleaves + 2] the same of rows (launch_list_rows)
  const float* sax_tab;  // [slot][16 x 256] the query's LB_SAX terms (k_query_prep), 16-byte aligned
  int cand_lo, cand_hi;  // candidates [cand_lo, cand_hi) of the sorted list; cand_hi <= 0: to the end
  const uint32_t* bound;  // [slot]
  uint32_t* list;         // [slot][list_stride] surviving rows
  uint64_t list_stride;
  uint32_t* list_count;   // [slot][8]: must be 0 before the launch
  unsigned long long* stats;  // [0] rows considered [2] rows pruned by LB_SAX [3] leaves visited
  int* err;                   // set to 1 when a bounded wait ran out (may be NULL)
};

// Stage 2: early-abandoning distances over a row list (or a row range).
struct EdArgs {
  const float* rows;  // leaf-ordered, row-major
  const int64_t* ids;
  int L;
  const uint32_t* list;        // [slot][list_stride] rows; NULL: the range below
  uint64_t list_stride;
  const uint32_t* list_count;  // [slot][8]
  const int* ident_leaf;       // [slot] range = this leaf's rows (device pointer), else
  uint64_t ident_first;        //   [ident_first, ident_first + ident_count)
  uint64_t ident_count;
  const uint64_t* leaf_start;
  const uint32_t* leaf_size;
  uint32_t min_batch;          // entries a warp takes at least, 1..32: with fewer in all, blocks stay idle
  uint32_t few_rows;           // one query over long rows: a warp each up to this many rows, 8 lanes each
                               // above (two launches); 0: 8 lanes, UINT32_MAX: a warp, whatever the count
  const float* q;              // [slot][L]
  int k;
  uint32_t* bound;             // [slot] float bits of the running k-th bound (atomicMin)
  uint32_t* kslots;            // [slot][kMaxK] distance bits: minima whose first k bound the k-th (atomicMin)
  unsigned long long* parts;   // [slot][parts_stride] per-block sorted lists (kWarpListCap stride)
  int* part_count;             // [slot][parts_stride]
  uint32_t parts_stride;       // lists per slot
  uint32_t period;             // turns between two looks at kslots by one warp (set by the launcher)
  unsigned long long* stats;   // [1] chunks computed [4] rows completed [5] rows started
  const int* gate;             // if set and *gate == 0, the launch scans nothing
  int has_floor;               // 1: only rows at distance > floor enter the lists (the
  float floor;                 //   answers of k above kMaxK come in rounds above it)
};

// Merge of a group's per-block lists into its running top-k, then either the
// candidate leaves of the next stage or the answers.
struct MergeArgs {
  const unsigned long long* parts;  // [slot][parts_stride][kWarpListCap]
  const int* part_count;            // [slot][parts_stride]
  uint32_t parts_stride;
  int nparts;
  int k;
  unsigned long long* topk;  // [slot][kMaxK]
  int* topk_count;           // [slot]
  uint32_t* bound;           // [slot]
  float* dist_out;           // [slot][k] answers; both NULL: none written
  int64_t* id_out;
  const uint32_t* out_row;   // [slot] row of the answers in dist_out / id_out; NULL: the slot
  uint32_t out_stride;       // entries per row with out_row
};

// Candidate leaves of a group (LB_EAPCA within the bound, in LB order).
struct SelectArgs {
  const float* lb;  // [slot][nleaves]
  int nleaves;
  const int* approx_leaf;  // [slot]
  const uint64_t* leaf_start;
  const uint32_t* leaf_size;
  int* cand;              // as in FilterArgs
  float* cand_lb;
  int* cand_count;
  uint32_t* unit_prefix;
  int by_file;            // leaves within a finite bound may stay in file order
  uint32_t* row_prefix;   // [slot][nleaves + 2] exclusive prefix of rows; NULL: not wanted
  uint32_t* gkeys;        // [slot][4 x nleaves], needed above kMaxLeavesSort leaves
};

int sm_count(int device);


// build
// node_of[r] = the leaf row first + r reaches in the tree, r < count
cudaError_t launch_route_rows(const float* X, int L, uint64_t first, uint32_t count, Tree t, int* node_of,
                              cudaStream_t s);
// The rows r < end of the leaves about to split: slot_of[node_of[r]] = p >= 0
// puts row r <= last[p] (a member of leaf p) into list[start[p] ..) and a
// later row (routed to it, not inserted yet) into list[members ..), in any
// order; counts[p] and *later (0 before the launch) count them.  Also resets
// the envelope keys of nsegs segments.
cudaError_t launch_collect_members(const int* node_of, uint64_t end, const int* slot_of, const uint64_t* start,
                                   const uint32_t* last, uint64_t members, uint32_t* list, uint32_t* counts,
                                   uint32_t* later, int* keys, int nsegs, cudaStream_t s);
// Segment envelopes of groups of rows: group g is rows start[g] .. + size[g],
// of members if set, and segments seg_off[g] .. seg_off[g + 1].
struct SketchArgs {
  const float* X;
  int L;
  const uint32_t* members;
  int ngroups;
  const uint64_t* start;
  const uint32_t* size;
  const int* seg_off;
  int max_segs;          // most segments of a group
  uint32_t max_size;     // most rows of a group
  const short* seg_from;
  const short* seg_to;
  int* keys;             // [segment][4] {max mean, min mean, max stdev, min stdev}, order-preserving ints
};
cudaError_t launch_sketch(const SketchArgs& a, cudaStream_t s);
// The redistribution of splits: node_of of the rows in list (`members` of
// them, then *later more) becomes a child of their leaf; n_left[p] (0 before
// the launch) counts the members of leaf p sent left.
struct SplitPolicy {
  float value;
  int left, right;
  short from, to;
  int idx;
};
cudaError_t launch_split_members(const float* X, int L, int* node_of, const uint32_t* list, uint64_t members,
                                 const uint32_t* later, uint64_t later_max, const int* slot_of, const SplitPolicy* splits,
                                 uint32_t* n_left, cudaStream_t s);
cudaError_t launch_widen_ids(const uint32_t* perm, uint64_t n, int64_t* ids, cudaStream_t s);
cudaError_t launch_gather_rows(const float* X, int L, const uint32_t* perm, uint64_t n, float* rows,
                               cudaStream_t s);
cudaError_t launch_sax_rows(const float* rows, int L, uint64_t n, const float* bp, uint8_t* sax,
                            cudaStream_t s);

// queries
cudaError_t launch_query_prep(const PrepArgs& a, int slots, cudaStream_t s);
cudaError_t launch_route_queries(const float* Q, int nq, int L, Tree t, int* leaf_out, cudaStream_t s,
                                 uint32_t* zero_a = nullptr, uint32_t na = 0, uint32_t* zero_b = nullptr,
                                 uint32_t nb = 0, unsigned long long* stamp = nullptr);
cudaError_t launch_pscan_prep(uint32_t* bound, uint32_t* kslots, int* topk_count, int slots, cudaStream_t s);
// blocks: per slot
cudaError_t launch_list_rows(const FilterArgs& a, int slots, int blocks, cudaStream_t s);
cudaError_t launch_lbsax_filter(const FilterArgs& a, int slots, int blocks, cudaStream_t s);
size_t lbsax_filter_smem();
// blocks: per slot, at most EdArgs::parts_stride
cudaError_t launch_ed_stream(const EdArgs& a, int slots, int blocks, cudaStream_t s);
// batched path: the (leaf, query) pairs whose LB_EAPCA is within the query's
// bound (k_leaf_keep)
cudaError_t launch_leaf_keep(const float* Q, int L, int nq, const short* useg_start, const short* useg_end, int nu,
                             float2* segstats, const int* seg_off, const short* points, const int* seg_uid,
                             const float* sk, const uint32_t* leaf_size, int nleaves, const float* bound,
                             uint32_t* leaf_cnt, uint32_t* leaf_q, uint32_t stride, cudaStream_t s);
// the same over the queries qlist[0 .. *nq_dev) (nq: their most), with the
// segment statistics already computed
cudaError_t launch_leaf_keep_list(const float2* segstats, int nu, int L, int nq, const int* seg_off,
                                  const short* points, const int* seg_uid, const float* sk, const uint32_t* leaf_size,
                                  int nleaves, const float* bound, uint32_t* leaf_cnt, uint32_t* leaf_q,
                                  uint32_t stride, const uint32_t* qlist, const uint32_t* nq_dev, cudaStream_t s);
// epsilon search: *flag = (lb <= stale / eps1), the reference's test of a
// candidate leaf against its k-th distance of that moment; *scanned counts
// the leaves that pass
cudaError_t launch_leaf_gate(float lb, float eps1, const uint32_t* stale, int* flag, unsigned long long* scanned,
                             cudaStream_t s);
// *stale = *bound when *flag
cudaError_t launch_stale_copy(const int* flag, const uint32_t* bound, uint32_t* stale, cudaStream_t s);
// resident blocks per SM of the distance stream for series length L
int ed_blocks_per_sm(int L);
// the same with id = row index (EdArgs::ids unused), blocks of 32 warps
cudaError_t launch_ed_stream_row_ids(const EdArgs& a, int slots, int blocks, cudaStream_t s);
cudaError_t launch_merge(const MergeArgs& a, int slots, cudaStream_t s);
// the merge, then the candidate selection against the merged bound
cudaError_t launch_merge_select(const MergeArgs& a, const SelectArgs& sel, int slots, cudaStream_t s);
cudaError_t launch_emit(const unsigned long long* topk, const int* topk_count, int k, float* dist_out,
                        int64_t* id_out, cudaStream_t s);

// data
// unit = 1: unit-normalised Gaussian rows / L2-normalised noisy queries
cudaError_t launch_generate_walks(uint64_t seed, uint64_t first, uint64_t n, int L, float* out,
                                  cudaStream_t s, int unit = 0);
cudaError_t launch_generate_queries(uint64_t seed, const float* data, uint64_t n, int L, int nq,
                                    const double* sigma2, float* out, uint64_t* base_ids, cudaStream_t s,
                                    int unit = 0, uint64_t data_seed = 0);  // data == nullptr: rows from data_seed

}  // namespace hg
