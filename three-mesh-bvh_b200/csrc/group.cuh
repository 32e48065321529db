// Group traversals: four neighbouring lanes share one query and walk the four-child records
// (layout.h), one child box or one triangle of a run per lane, so that a step's chain of dependent
// instructions is that of one box or one triangle.  All shuffles and ballots are whole-warp ones in
// convergent code; a group that has nothing to do in a step is masked.
//
// The stack of a group is in shared memory (link and entry distance per entry, `cap` entries; the
// host sizes it to the tree, MeshDev::quad_stack), one entry of padding apart from the next group's so
// that the eight groups' equal depths fall into different banks.
#pragma once

#include "traverse.cuh"

namespace bvhc {
namespace dev {

constexpr int kGroup = 4;                        // lanes per query
constexpr int kGroups = 32 / kGroup;             // queries per warp
constexpr int kBlockGroups = kBlock / kGroup;    // queries per block

// The smallest of a group's four values, in every lane.
__device__ __forceinline__ float group_min(float v) {
  v = fminf(v, __shfl_xor_sync(0xFFFFFFFFu, v, 1));
  return fminf(v, __shfl_xor_sync(0xFFFFFFFFu, v, 2));
}

// Order of a group's children: `key` is a float's bits with the lane in the low two bits, or
// 0x7FFFFFFF for a child that is not entered, compared as signed integers (negative distances, boxes
// that hold the origin, come first in any order).  rank: how many children come before this lane's;
// first: the lane (0..3) of the nearest one.
__device__ __forceinline__ void group_rank(int key, int& rank, unsigned& first) {
  const unsigned full = 0xFFFFFFFFu;
  const int a = __shfl_xor_sync(full, key, 1), b = __shfl_xor_sync(full, key, 2), c = __shfl_xor_sync(full, key, 3);
  rank = (a < key) + (b < key) + (c < key);
  first = (unsigned)__vimin3_s32(__vimin3_s32(key, a, b), c, c) & 3u;
}

}  // namespace dev

static inline size_t group_smem(int stack) { return (size_t)dev::kBlockGroups * (stack + 1) * sizeof(uint2); }

}  // namespace bvhc
