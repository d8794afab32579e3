// hg_items.h -- sizes that the host's buffers and the kernels that fill them
// must agree on.  No CUDA in here: a CPU test holds one against the other.
#pragma once

#include <stdint.h>

#include "hg_arith.cuh"  // HG_HD

namespace hg {

constexpr int kBatchBoundQueries = 64;  // queries per tile in the bound pass (MMA N = 64)

// Work items that even out over the SMs: the filter's work lists are cut into
// at least this many items where their tiles allow it
constexpr uint32_t kBatchItemTarget = 8 * 148;

// The bound pass's work list holds, for every group of at most
// kBatchBoundQueries queries of one leaf, the leaf's tiles in chunks.  Room for
// any batch of nq queries over `leaves` leaves of at most max_use tiles: chunks
// of btpi tiles, and what shorter chunks (bound_item_tiles) add.  Of b =
// max(2, floor(work / kBatchItemTarget)) tiles there are work / b, fewer than 1.5
// kBatchItemTarget (most for work just below 3 kBatchItemTarget), and at most one
// more per group, of which there are at most nq.
inline uint64_t bound_items_room(uint32_t nq, uint64_t leaves, uint32_t max_use, uint32_t btpi) {
  const uint64_t groups = ((uint64_t)nq + kBatchBoundQueries - 1) / kBatchBoundQueries + leaves;
  return groups * ((max_use + btpi - 1) / btpi) + 2 * kBatchItemTarget + nq;
}

// Tiles per item for `work` (group, tile) pairs in `groups` groups: btpi, or
// fewer, down to 2, until there are kBatchItemTarget items -- where that list
// fits `room` items (it does in room of bound_items_room).
HG_HD uint32_t bound_item_tiles(uint64_t work, uint64_t groups, uint32_t btpi, uint64_t room) {
  const uint64_t even = work / kBatchItemTarget, b = even > 2 ? even : 2;
  return b < btpi && work / b + groups <= room ? (uint32_t)b : btpi;
}

constexpr uint32_t kBatchPairBlock = 1024;  // survivor pairs a filter warp reserves at a time
constexpr uint32_t kBatchPairWarps = 8;     // filter warps per SM that do

// The block of the pair list (pairs_cap slots) that a filter warp got for the
// counter's value nb: slots [*cur, *end).  Past the list's end *cur is
// pairs_cap + 1, and the warp reserves no more: the counter then says that pairs
// were lost, and ends within a block per warp of that.  (A warp that went on
// took 1,024 counts for every 32 survivors it dropped: 134M of them wrapped the
// counter, and the list could look whole.)
HG_HD void pair_block(uint32_t nb, uint32_t pairs_cap, uint32_t* cur, uint32_t* end) {
  *cur = nb < pairs_cap ? nb : pairs_cap + 1;
  *end = nb + kBatchPairBlock < pairs_cap ? nb + kBatchPairBlock : (nb < pairs_cap ? pairs_cap : pairs_cap + 1);
}
HG_HD bool pair_list_full(uint32_t cur, uint32_t pairs_cap) { return cur > pairs_cap; }

}  // namespace hg
