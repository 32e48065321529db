// What the closestPointToPoint kernels and the shapecast queries share: the distance to a box and the
// maxThreshold test on it, and the phased kernel's launch.
#pragma once

#include <cfloat>

#include "group.cuh"

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

constexpr uint32_t kNoRecord = 0xFFFFFFFFu;

// Float32 closest point of a triangle: closest_sq_f's regions (Ericson, Real-Time Collision Detection,
// 5.1.5) as selections of two numerators over one denominator, l = ab v + ac w, and one reciprocal:
// the lanes of a warp are at different triangles, and would walk the regions' branches, and their
// divisions, one after the other.
struct Candidate {
  float d2, err;
  float3 q;
};
__device__ __forceinline__ Candidate candidate(float3 p, const Tri& t) {
  const float abx = t.b.x - t.a.x, aby = t.b.y - t.a.y, abz = t.b.z - t.a.z;
  const float acx = t.c.x - t.a.x, acy = t.c.y - t.a.y, acz = t.c.z - t.a.z;
  const float apx = p.x - t.a.x, apy = p.y - t.a.y, apz = p.z - t.a.z;
  const float sc = max3(fabsf(abx), fabsf(aby), fabsf(abz)) + max3(fabsf(acx), fabsf(acy), fabsf(acz)) +
                   max3(fabsf(apx), fabsf(apy), fabsf(apz));
  const float d1 = abx * apx + aby * apy + abz * apz;
  const float d2 = acx * apx + acy * apy + acz * apz;
  const float bpx = apx - abx, bpy = apy - aby, bpz = apz - abz;
  const float d3 = abx * bpx + aby * bpy + abz * bpz;
  const float d4 = acx * bpx + acy * bpy + acz * bpz;
  const float cpx = apx - acx, cpy = apy - acy, cpz = apz - acz;
  const float d5 = abx * cpx + aby * cpy + abz * cpz;
  const float d6 = acx * cpx + acy * cpy + acz * cpz;
  const float e43 = d4 - d3, e56 = d5 - d6;
  // both are zero where b = c, a segment, which is met on its edge a b: the products' fused difference is not
  const float vc = e43 == 0.0f && e56 == 0.0f ? 0.0f : d1 * d4 - d3 * d2;
  const float vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
  // the first region that holds wins, so they are taken last to first
  float nv = vb, nw = vc, den = va + vb + vc;
  const bool bc = va <= 0.0f && e43 >= 0.0f && e56 >= 0.0f;
  den = bc ? e43 + e56 : den;
  nv = bc ? e56 : nv;
  nw = bc ? e43 : nw;
  const bool ac = vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f;
  den = ac ? d2 - d6 : den;
  nv = ac ? 0.0f : nv;
  nw = ac ? d2 : nw;
  const bool at_c = d6 >= 0.0f && d5 <= d6;
  den = at_c ? 1.0f : den;
  nv = at_c ? 0.0f : nv;
  nw = at_c ? 1.0f : nw;
  const bool ab = vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f;
  den = ab ? d1 - d3 : den;
  nv = ab ? d1 : nv;
  nw = ab ? 0.0f : nw;
  const bool at_b = d3 >= 0.0f && d4 <= d3, at_a = d1 <= 0.0f && d2 <= 0.0f;
  den = at_a || at_b ? 1.0f : den;
  nv = at_a ? 0.0f : at_b ? 1.0f : nv;
  nw = at_a || at_b ? 0.0f : nw;
  const float rd = rcp_fast(den), v = nv * rd, w = nw * rd;
  const float lx = abx * v + acx * w, ly = aby * v + acy * w, lz = abz * v + acz * w;
  const float rx = apx - lx, ry = apy - ly, rz = apz - lz;
  Candidate c;
  c.d2 = rx * rx + ry * ry + rz * rz;
  const float e = 32.0f * kU * sc;  // |error| of each closest-point coordinate (local-frame evaluation)
  float root;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"(c.d2));
  c.err = 3.501f * e * root + 3.0f * e * e;
  const bool vb_ = !at_a && at_b, vc_ = !at_a && !at_b && !ab && at_c;
  c.q.x = vb_ ? t.b.x : vc_ ? t.c.x : t.a.x + lx;
  c.q.y = vb_ ? t.b.y : vc_ ? t.c.y : t.a.y + ly;
  c.q.z = vb_ ? t.b.z : vc_ ? t.c.z : t.a.z + lz;
  return c;
}

// Which vertex of the triangle q is, bit for bit (3: none).
__device__ __forceinline__ uint32_t vertex_of(const Tri& t, float3 q) {
  return q.x == t.a.x && q.y == t.a.y && q.z == t.a.z   ? 0u
         : q.x == t.b.x && q.y == t.b.y && q.z == t.b.z ? 1u
         : q.x == t.c.x && q.y == t.c.y && q.z == t.c.z ? 2u
                                                        : 3u;
}

// Whether the triangle's box is farther than the best candidate for certain: at most 4 roundings above
// the exact value's relative 2^-22, so the 2^-20 shrink keeps the distance a lower bound.
__device__ __forceinline__ bool beyond(float3 p, const Tri& t, float best_hi) {
  const float dx = fmaxf(fmaxf(fminf(t.a.x, fminf(t.b.x, t.c.x)) - p.x, p.x - fmaxf(t.a.x, fmaxf(t.b.x, t.c.x))), 0.0f);
  const float dy = fmaxf(fmaxf(fminf(t.a.y, fminf(t.b.y, t.c.y)) - p.y, p.y - fmaxf(t.a.y, fmaxf(t.b.y, t.c.y))), 0.0f);
  const float dz = fmaxf(fmaxf(fminf(t.a.z, fminf(t.b.z, t.c.z)) - p.z, p.z - fmaxf(t.a.z, fmaxf(t.b.z, t.c.z))), 0.0f);
  return (dx * dx + dy * dy + dz * dz) * (1.0f - 0x1p-20f) > best_hi;
}

// A lane's best candidate: float32 squared distance and its error bound, the triangle record with its
// vertex above kRunShift, its faceIndex and the float32 closest point; and the candidates that float32
// cannot tell from it (`ties` of them, in the lane's column of a shared array).
struct Nearest {
  float d2, err;
  uint32_t rec, face;
  float3 q;
  int ties;
};
__device__ __forceinline__ Nearest nearest_none() {
  return {kInf, 0.0f, kNoRecord, 0u, make_float3(0.f, 0.f, 0.f), 0};
}

// A candidate whose float32 closest point is 0 / 0, or may be.  Where the first two corners coincide (a zero
// denominator on their edge) it is in the reference's arithmetic too, unless another region is nearest, and
// the reference then does not take the triangle: d2 is not a number.  Elsewhere float32 has underflowed.
static __device__ __noinline__ Candidate candidate_slow(float3 p, float3 a, float3 b, float3 c) {
  const CPFF e = closest_ff(p, a, b, c);
  Candidate r;
  r.d2 = e.d2.hi;
  r.err = fabsf(e.d2.hi) * 0x1p-40f + 1e-37f;
  r.q = make_float3(ff_to_f(e.q.x), ff_to_f(e.q.y), ff_to_f(e.q.z));
  return r;
}
__device__ __forceinline__ bool no_first_edge(const Tri& t) {
  return t.a.x == t.b.x && t.a.y == t.b.y && t.a.z == t.b.z;
}

// Whether squared distance d of faceIndex fd goes before e of fe: nearer, or an exact tie and the smaller
// faceIndex.  What is not a number goes before nothing.
__device__ __forceinline__ bool nearer(ff d, uint32_t fd, ff e, uint32_t fe) {
  return ff_lt(d, e) || (d.hi == e.hi && d.lo == e.lo && fd < fe) || (e.hi != e.hi && d.hi == d.hi);
}

// Whether candidate `cand` beats `b` where their float32 distances do not tell: the same vertex is an
// exact tie, else the float-float distances decide; an exact tie goes to the smaller faceIndex.
static __device__ __noinline__ bool closer_slow(const TriRecord* __restrict__ tris, float3 p, uint32_t cand,
                                                uint32_t b) {
  const Tri t = load_tri(tris, cand & kRunFirst), u = load_tri(tris, b & kRunFirst);
  const uint32_t tv = cand >> kRunShift, uv = b >> kRunShift;
  if (tv != 3u && uv != 3u && same_vertex(t, tv, u, uv)) return t.face < u.face;
  return nearer(closest_ff(p, t.a, t.b, t.c).d2, t.face, closest_ff(p, u.a, u.b, u.c).d2, u.face);
}

// Offers triangle t (record k) at candidate c to a lane's best.  Candidates are ranked by exact distance,
// then by faceIndex, a total order that does not depend on the order of the offers.  What float32 and
// the shared vertex do not settle is kept beside the best one for the finalize kernel: most of it is
// overtaken by a nearer triangle later in the walk, and float-float code in the loop is fetched and
// executed by whole warps for one lane.
__device__ __forceinline__ void offer_closest(const TriRecord* __restrict__ tris, float3 p, const Tri& t, uint32_t k,
                                              Candidate c, Nearest& b, uint2 (*s_tie)[kBlock]) {
  if (c.d2 - c.err > b.d2 + b.err) return;
  if (no_first_edge(t) || c.d2 != c.d2) {
    c = candidate_slow(p, t.a, t.b, t.c);
    if (!(c.d2 < kInf)) return;
  }
  const float hi = c.d2 + c.err, lo = c.d2 - c.err;
  bool take = b.rec == kNoRecord ? c.d2 < kInf : hi < b.d2 - b.err;
  uint32_t rec = kNoRecord;
  if (!take && b.rec != kNoRecord && !(lo > b.d2 + b.err)) {
    rec = k | vertex_of(t, c.q) << kRunShift;
    if ((rec >> kRunShift) != 3u && (b.rec >> kRunShift) != 3u && c.q.x == b.q.x && c.q.y == b.q.y && c.q.z == b.q.z) {
      take = t.face < b.face;  // the same vertex: an exact tie, the smaller faceIndex wins
    } else if (b.ties < kClosestTies) {
      take = c.d2 < b.d2;
      s_tie[b.ties][threadIdx.x] = take ? make_uint2(b.rec, __float_as_uint(b.d2 - b.err))
                                        : make_uint2(rec, __float_as_uint(lo));
      ++b.ties;
    } else {
      take = closer_slow(tris, p, rec, b.rec);
    }
  }
  if (take) {
    b.d2 = c.d2;
    b.err = c.err;
    b.rec = rec != kNoRecord ? rec : k | vertex_of(t, c.q) << kRunShift;
    b.face = t.face;
    b.q = c.q;
    int kept = 0;  // ties that the new best candidate leaves behind for certain are dropped
    for (int j = 0; j < b.ties; ++j) {
      const uint2 e = s_tie[j][threadIdx.x];
      if (!(__uint_as_float(e.y) > hi)) s_tie[kept++][threadIdx.x] = e;
    }
    b.ties = kept;
  }
}

// The box of a record's child against maxThreshold^2, exactly.
static __device__ __noinline__ bool under_max_slow(const BoxChild* c, float3 p, ff max2) {
  const float b[6] = {c->lo[0], c->lo[1], c->lo[2], c->hi[0], c->hi[1], c->hi[2]};
  return ff_lt(box_score_ff(b, p), max2);
}

// The record of a query whose walk G neighbouring lanes shared (4, or the whole warp), from the lanes'
// best candidates: the nearest with what is not settled against it, five words for
// closest_point_finalize_kernel.  Called by whole warps; groups with `on` false write nothing.
template <int G>
__device__ __forceinline__ void store_merged(const TriRecord* __restrict__ tris, float3 p, const Nearest& best, bool on,
                                             uint32_t* o, uint2 (*s_tie)[kBlock]) {
  const unsigned full = 0xFFFFFFFFu, lane = threadIdx.x & 31u, base = lane & ~(G - 1u), j = lane & (G - 1u);
  const unsigned group = G == 32 ? full : ((1u << (G & 31)) - 1u);
  int key = best.rec == kNoRecord ? 0x7FFFFFFF : (int)((__float_as_uint(best.d2) & ~(G - 1u)) | j);
#pragma unroll
  for (int x = 1; x < G; x <<= 1) key = min(key, __shfl_xor_sync(full, key, x));
  const unsigned src = base + ((unsigned)key & (G - 1u));
  const float hi = __shfl_sync(full, best.d2 + best.err, src);
  uint32_t rec = __shfl_sync(full, best.rec, src);
  const float qx = __shfl_sync(full, best.q.x, src), qy = __shfl_sync(full, best.q.y, src),
              qz = __shfl_sync(full, best.q.z, src);
  bool extra = lane != src && best.rec != kNoRecord && !(best.d2 - best.err > hi);
  const bool same = extra && (rec >> kRunShift) != 3u && (best.rec >> kRunShift) != 3u && best.q.x == qx &&
                    best.q.y == qy && best.q.z == qz;
  extra = extra && !same;
  // of the lanes at the same vertex the smallest faceIndex
  uint32_t f = same || lane == src ? best.face : 0xFFFFFFFFu;
#pragma unroll
  for (int x = 1; x < G; x <<= 1) f = min(f, __shfl_xor_sync(full, f, x));
  const unsigned winner = (__ballot_sync(full, (same || lane == src) && best.face == f) >> base) & group;
  rec = __shfl_sync(full, best.rec, base + (unsigned)__ffs(winner) - 1u);
  int mine = extra ? 1 : 0;
  for (int k = 0; k < best.ties; ++k) mine += !(__uint_as_float(s_tie[k][threadIdx.x].y) > hi);
  if (!on || best.rec == kNoRecord) mine = 0;
  int at = mine;  // inclusive prefix within the group
#pragma unroll
  for (int x = 1; x < G; x <<= 1) {
    const int y = __shfl_up_sync(full, at, x);
    if ((int)j >= x) at += y;
  }
  const int total = __shfl_sync(full, at, base + G - 1u);
  at -= mine;
  const bool over = on && total > kClosestTies;  // more than the record holds: settled here
  if (__ballot_sync(full, over)) {
    uint32_t r = best.rec;
    if (over && r != kNoRecord)
      for (int k = 0; k < best.ties; ++k)
        if (closer_slow(tris, p, s_tie[k][threadIdx.x].x, r)) r = s_tie[k][threadIdx.x].x;
#pragma unroll 1
    for (int x = 1; x < G; x <<= 1) {
      const uint32_t c = __shfl_xor_sync(full, r, x);
      if (over && c != kNoRecord && (r == kNoRecord || closer_slow(tris, p, c, r))) r = c;
    }
    if (over) {
      rec = r;
      mine = 0;
    }
  }
  if (!on) return;
  if (j == 0) {
    o[0] = rec;
    o[1] = over ? 0u : (uint32_t)total;
  }
  if (mine) {
    if (extra) o[2 + at++] = best.rec;
    for (int k = 0; k < best.ties; ++k)
      if (!(__uint_as_float(s_tie[k][threadIdx.x].y) > hi)) o[2 + at++] = s_tie[k][threadIdx.x].x;
  }
}

// A child's box (its squared distance from p in `s`) against the bound reached and maxThreshold: parts of
// leaves, whose boxes the reference does not have, only against the bound.
struct MaxThreshold {
  ff max2;
  float lo, hi;  // distances outside [lo, hi) are decided by their float32 value (see under_max)
};
__device__ __forceinline__ MaxThreshold max_threshold(float max_t) {
  const ff m = two_prod(max_t, max_t);
  return {m, m.hi * (1.0f - kSlabMargin) * (1.0f - 0x1p-19f), m.hi * (1.0f + 0x1p-18f)};
}
__device__ __forceinline__ bool box_wanted(const BoxChild* __restrict__ c, float3 p, float bound, const MaxThreshold& mx,
                                           float& s, uint32_t& link) {
  float4 a, b;
  ld8(c, a, b);
  link = __float_as_uint(b.z);
  const float dx = max3(a.x - p.x, p.x - a.w, 0.0f), dy = max3(a.y - p.y, p.y - b.x, 0.0f),
              dz = max3(a.z - p.z, p.z - b.y, 0.0f);
  s = dx * dx + dy * dy + dz * dz;
  if (!(s <= bound)) return false;
  if (s < mx.lo || __float_as_uint(b.w) != 0u) return true;
  return s < mx.hi && under_max_slow(c, p, mx.max2);
}

// A query's walk by its whole warp, `sp` stacked entries (squared distance and link) under `root`: the lanes'
// best candidates.
__device__ __forceinline__ void closest_walk_wide(const MeshDev& m, float3 p, const MaxThreshold& mx, uint2* stack,
                                                  int spare, int sp, int root, float bound, Nearest& best,
                                                  uint2 (*s_tie)[kBlock]) {
  const unsigned full = 0xFFFFFFFFu, lane = threadIdx.x & 31u, j = lane & 3u;
  for (;;) {
    while (sp > 0) {
      WideEntry e = wide_take(stack, sp, lane, spare);
      e.on = e.on && e.key <= bound;
      const bool leaf = e.on && (e.link & kLeafBit);
      bool enter = false;
      uint32_t link = 0u;
      float key = 0.0f;
      if (e.on && !leaf) {
        const BoxChild* c = m.boxes[e.link].c + j;
        enter = box_wanted(c, p, bound, mx, key, link);
      }
      if (leaf && j <= ((e.link >> kRunShift) & 3u)) {
        const uint32_t k = (e.link & kRunFirst) + j;
        const Tri t = load_tri(m.tris, k);
        offer_closest(m.tris, p, t, k, candidate(p, t), best, s_tie);
      }
      if (__ballot_sync(full, leaf))
        bound = fminf(bound, warp_min(fminf((best.d2 + best.err) * (1.0f + 0x1p-18f), FLT_MAX)));
      if (__ballot_sync(full, enter)) wide_push(stack, sp, lane, enter, link, key, key);
    }
    if (++root >= m.n_roots) return;
    sp = 1;
    if (lane == 0) stack[0] = make_uint2(m.quad_roots[root], 0u);
    __syncwarp();
  }
}

}  // namespace dev

// Up to this many queries take the whole warp each (kernels_wide.cu), more four lanes, the last of a warp again
// all 32.  A query about as far from many triangles (on the axis of a tube) walks hundreds of steps after the
// others are done, and the whole warp takes up to eight of them at once; a query near the surface is done in a
// few, and the whole warp is wasted on it.  So the line depends on the queries, and on how long walks are.
// 80,000-triangle knot, points about the surface, seven tenths of them so and the rest spread, all spread, a grid:
// 32,000 points 200, 265, 331, 278 us by warps (four lanes 120, 304, 413, 445), 70,000 points 359, 484, 624, 462
// (185, 490, 652, 714), 100,000 points 507, 650, 863, 628 (234, 503, 751, 802).  10,000 triangles: 16,000 points
// 93, 106, 128, 97 (81, 114, 167, 155), 32,000 points 157, 183, 204, 165 (97, 148, 183, 194), 70,000 points
// 288, 329, 388, 285 (144, 218, 292, 269).
// Odd variants without tiles, which are for coherent queries, take the shared traversal in input order beyond this
// many: grids on the 80,000-triangle knot, 140,000 points 1.25 ms shared (four lanes 1.06), 195,112 1.25 (1.10),
// 300,000 1.37 (1.60), 2,097,152 4.1 (8.7), 16,777,216 21 (61).
constexpr uint64_t kSharedQueries = 200000;
static inline uint32_t wide_queries(const MeshDev& m) { return m.n_tris < 50000 ? 32768 : 65536; }
cudaError_t launch_closest_wide(const MeshDev& m, const float* pts, uint32_t n, float max_t, bvhc_closest* out,
                                cudaStream_t stream);

// closestPointToPoint's traversals with minThreshold 0 (kernels_closest.cu): pending records of five words
// (triangle record and vertex, or 0xFFFFFFFF; number of undecided candidates; those).  shared: the 32 queries of
// a warp in one traversal of the child pairs (m.n_tris < kRunFirst), in the order of `queue` (nullable), or with
// pitch > 0 in tiled order with 2^rows_log2 rows a tile; else over the four-child records (group_stack(m) > 0).
cudaError_t launch_closest_phased(const MeshDev& m, const float* pts, uint32_t n, float max_t, bvhc_closest* out,
                                  bool shared, const uint32_t* queue, uint32_t pitch, int rows_log2,
                                  cudaStream_t stream);

}  // namespace bvhc
