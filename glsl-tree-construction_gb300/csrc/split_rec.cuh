// split_rec.cuh - what the radix tree kernel leaves per split for the octree
// kernel (octree_window.cuh): one word each, in split order.
//
// The node whose split is x covers the keys [lo, hi].  Near splits (both ends
// within SPLIT_FAR positions) carry, from bit 30 down: octree nodes owned (5
// bits: the edge count, SPLIT_ROOT for the root), depth (5), whether the node
// is its parent's left child (1), x - lo (10), hi - x (10).  The parent's
// split is hi for a left child and lo - 1 for a right one, and the node's
// Karras index is hi or lo.  Far splits have bit 31 set and carry the Karras
// index; SPLIT_NONE is no split (a cloud's last key).
#pragma once

#include <stdint.h>

namespace gtc {

constexpr int SPLIT_FAR = 1024;
constexpr uint32_t SPLIT_FAR_FLAG = 1u << 31, SPLIT_NONE = ~0u;
constexpr uint32_t SPLIT_ROOT = 31u;  // more than any edge count (at most 21)

__device__ __forceinline__ uint32_t split_pack(uint32_t x, uint32_t lo, uint32_t hi, uint32_t kidx, uint32_t owned,
                                               uint32_t depth, bool left_child) {
  if (x - lo >= (uint32_t)SPLIT_FAR || hi - x >= (uint32_t)SPLIT_FAR) return SPLIT_FAR_FLAG | kidx;
  return (owned << 26) | (depth << 21) | ((left_child ? 1u : 0u) << 20) | ((x - lo) << 10) | (hi - x);
}
__device__ __forceinline__ bool split_far(uint32_t r) { return (r & SPLIT_FAR_FLAG) != 0; }  // or none
__device__ __forceinline__ uint32_t split_owned(uint32_t r) { return r >> 26; }
__device__ __forceinline__ bool split_root(uint32_t r) { return (r >> 26) == SPLIT_ROOT; }
__device__ __forceinline__ uint32_t split_depth(uint32_t r) { return (r >> 21) & 31u; }
__device__ __forceinline__ int split_lo(uint32_t r) { return (int)((r >> 10) & 1023u); }
__device__ __forceinline__ int split_hi(uint32_t r) { return (int)(r & 1023u); }
// Relative to the split: the Karras index, and the parent's split.
__device__ __forceinline__ int split_kidx(uint32_t r) { return (r >> 20) & 1u ? split_hi(r) : -split_lo(r); }
__device__ __forceinline__ int split_parent(uint32_t r) { return (r >> 20) & 1u ? split_hi(r) : -split_lo(r) - 1; }

}  // namespace gtc
