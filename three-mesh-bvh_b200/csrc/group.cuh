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

// ---------------------------------------------------------------------------------------------
// A warp takes the up to eight newest entries of its stack at once, four lanes each: an entry that is a
// record has its four children tested, one that is a run its triangles.  What is entered goes back on
// the stack, the newest entry's children on top, nearest first.  A step tests what eight steps of a
// single walk would; some of it the nearer entries' results would have spared, which costs nothing
// while the chip is otherwise idle.
// Stack: `cap` entries per warp.  Eight entries are taken while what they can add (32) and one depth-
// first walk (quad_stack) still fit above the rest, else one, so nothing overflows.
// ---------------------------------------------------------------------------------------------
constexpr int kWideSpare = 256;
__host__ __device__ inline int wide_stack(int quad_stack) { return kWideSpare + 32 + quad_stack; }

struct WideEntry {
  uint32_t link;
  float key;
  bool on;
};
// This lane's group's entry, and the stack without what was taken.
__device__ __forceinline__ WideEntry wide_take(const uint2* stack, int& sp, unsigned lane, int spare = kWideSpare) {
  const int width = sp <= spare ? 8 : 1, g = (int)(lane / kGroup);
  WideEntry e{0u, 0.0f, g < width && g < sp};
  if (e.on) {
    const uint2 v = stack[sp - 1 - g];
    e.link = v.x;
    e.key = __uint_as_float(v.y);
  }
  sp -= min(width, sp);
  __syncwarp();
  return e;
}
// Stacks the children that are entered: the first group's on top, each group's nearest first.
__device__ __forceinline__ void wide_push(uint2* stack, int& sp, unsigned lane, bool enter, uint32_t link, float key,
                                          float word) {
  const unsigned full = 0xFFFFFFFFu, j = lane & 3u, base = lane & ~3u;
  int rank;
  unsigned first;
  group_rank(enter ? (int)((__float_as_uint(key) & ~3u) | j) : 0x7FFFFFFF, rank, first);
  const unsigned all = __ballot_sync(full, enter);
  if (enter) {
    const int later = base == 28u ? 0 : __popc(all >> (base + kGroup)), own = __popc((all >> base) & 0xFu);
    stack[sp + later + own - 1 - rank] = make_uint2(link, __float_as_uint(word));
  }
  sp += __popc(all);
  __syncwarp();
}
__device__ __forceinline__ float warp_min(float v) {
  for (int x = 1; x < 32; x <<= 1) v = fminf(v, __shfl_xor_sync(0xFFFFFFFFu, v, x));
  return v;
}

}  // namespace dev

// Shared memory of a block's stacks: four lanes a query, or a warp.
static inline size_t group_smem(int stack) { return (size_t)dev::kBlockGroups * (stack + 1) * sizeof(uint2); }

static inline size_t wide_smem(int stack) { return (size_t)dev::kWarps * dev::wide_stack(stack) * sizeof(uint2); }

}  // namespace bvhc
