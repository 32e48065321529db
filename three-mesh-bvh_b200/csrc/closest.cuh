// What the closestPointToPoint kernels and the shapecast queries share: the distance to a box and the
// maxThreshold test on it, and the phased kernel's launch.
#pragma once

#include "traverse.cuh"

namespace bvhc {
namespace dev {

constexpr float kU = 5.9604644775390625e-08f;  // 2^-24

__device__ __forceinline__ float box_score(const float* b, float3 p) {
  float dx = fmaxf(b[0], fminf(b[3], p.x)) - p.x;
  float dy = fmaxf(b[1], fminf(b[4], p.y)) - p.y;
  float dz = fmaxf(b[2], fminf(b[5], p.z)) - p.z;
  return dx * dx + dy * dy + dz * dz;
}

static __device__ __noinline__ ff box_score_ff(const float* b, float3 p) {
  ff dx = two_diff(fmaxf(b[0], fminf(b[3], p.x)), p.x);
  ff dy = two_diff(fmaxf(b[1], fminf(b[4], p.y)), p.y);
  ff dz = two_diff(fmaxf(b[2], fminf(b[5], p.z)), p.z);
  return ff_add(ff_add(ff_mul(dx, dx), ff_mul(dy, dy)), ff_mul(dz, dz));
}

// score < maxThreshold^2, decided exactly (the box score carries at most 5 roundings, all terms
// positive, so 2^-20 relative slack separates every case the float32 value can settle).
__device__ __forceinline__ bool under_max(float s, const float* b, float3 p, ff max2) {
  if (s * (1.0f + kSlabMargin) < max2.hi * (1.0f - kSlabMargin)) return true;
  if (s * (1.0f - kSlabMargin) > max2.hi * (1.0f + kSlabMargin)) return false;
  return ff_lt(box_score_ff(b, p), max2);
}

// Candidates that float32 cannot tell apart are kept as a triangle record with, above kRunShift, the
// vertex that the float32 closest point is bit for bit (3: none).
constexpr int kClosestTies = 3;  // undecided candidates a traversal may leave beside its best one

__device__ __forceinline__ bool same_vertex(const Tri& t, uint32_t tv, const Tri& u, uint32_t uv) {
  const float3 v = tv == 0u ? t.a : tv == 1u ? t.b : t.c, w = uv == 0u ? u.a : uv == 1u ? u.b : u.c;
  return v.x == w.x && v.y == w.y && v.z == w.z;
}

}  // namespace dev

// closestPointToPoint's traversal over the four-child records, minThreshold 0 (kernels_closest.cu):
// pending records of five words (triangle record and vertex, or 0xFFFFFFFF; number of undecided
// candidates; those).  queue (nullable): the queries' order; pitch > 0:
// tiled order with 2^rows_log2 rows a tile.
cudaError_t launch_closest_phased(const MeshDev& m, const float* pts, uint32_t n, float max_t, bvhc_closest* out,
                                  const uint32_t* queue, uint32_t pitch, int rows_log2, cudaStream_t stream);

}  // namespace bvhc
