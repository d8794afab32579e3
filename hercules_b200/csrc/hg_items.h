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
// of btpi tiles, and what shorter chunks (bound_item_tiles) add.  Those have
// work / b tiles each for b = max(2, floor(work / kBatchItemTarget)), fewer than
// 1.5 kBatchItemTarget chunks (work just below 3 kBatchItemTarget), and one
// partly filled per group, of which there are at most nq.
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

}  // namespace hg
