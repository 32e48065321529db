// Device helpers shared by the traversal kernels (kernels_*.cu): rays, child-pair and triangle
// records, the conservative slab test, the raycastFirst leaf step and reported record, and the
// child order.  Each kernel is defined in exactly one translation unit; these helpers are inline
// device code and compile into each unit that uses them.
//
// One ray or query per thread (or per warp lane of a shared traversal).  Each visit of an internal
// node reads one 64-byte child-pair record (both child boxes and links) with four 16-byte
// read-only loads; each leaf is a contiguous run of 48-byte triangle records.  Traversal stacks are
// bounded (the mesh upload rejects deeper trees), and an overflow sets the device error word
// instead of faulting.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "kernels.cuh"
#include "raykey.cuh"
#include "robust.cuh"
#include "softf64.cuh"

namespace bvhc {
namespace dev {

constexpr int kBlock = 128;
constexpr int kWarps = kBlock / 32;
constexpr float kInf = __builtin_huge_valf();
constexpr float kSlabMargin = 9.5367431640625e-07f;  // 2^-20, relative slack on slab distances
constexpr float kTiny = 1e-30f;                      // stand-in for a zero direction component

__device__ __forceinline__ float4 ld4(const void* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
// 32 bytes in one load instruction (the 256-bit global load of sm_100) through the read-only path;
// p must be 32-byte aligned.
__device__ __forceinline__ void ld8(const void* p, float4& a, float4& b) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// Reciprocal within one unit in the last place; the slab margins absorb it.
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct RayF {
  float3 o, d, inv;
  float dk;  // kFilterK |d|_1 (tri_filter)
};

// 1 / direction.  A zero component is replaced by +-1e-30 so that (bound - origin) * inv is never 0 * inf:
// the slab then becomes (-huge, +huge) or empty, which is what the reference's NaN guards in
// intersectsNodeBounds (intersectUtils.js:52-54,70-72) amount to.  Any number serves that is large enough
// that a box's planes are behind or far ahead, and from an origin far out it is 2^126 / |o|, so that
// origin * inv stays finite.
// RARE: behind one branch, which suits the kernels that make a ray once; where one is made at every instance
// the selections cost less (1,048,576 rays over 512 instances 1.69 ms, with the branch 1.72).
template <bool RARE = true>
__device__ __forceinline__ float3 ray_reciprocals(float3 o, float3 d) {
  auto stand_in = [](float a, float b) {
    return fabsf(b) < kTiny ? copysignf(fmaxf(fminf(fabsf(a) * 0x1p-126f, 8.0f), kTiny), b) : b;
  };
  if (!RARE || min3(fabsf(d.x), fabsf(d.y), fabsf(d.z)) < kTiny)
    d = make_float3(stand_in(o.x, d.x), stand_in(o.y, d.y), stand_in(o.z, d.z));
  return make_float3(rcp_fast(d.x), rcp_fast(d.y), rcp_fast(d.z));
}

template <bool RARE = true>
__device__ __forceinline__ RayF make_ray(const float* __restrict__ rays, uint64_t i) {
  const float2* p = reinterpret_cast<const float2*>(rays + 6 * i);
  // rays are read once: streaming loads keep them from evicting the BVH from L2
  float2 r0 = __ldcs(p), r1 = __ldcs(p + 1), r2 = __ldcs(p + 2);
  RayF r;
  r.o = make_float3(r0.x, r0.y, r1.x);
  r.d = make_float3(r1.y, r2.x, r2.y);
  r.inv = ray_reciprocals<RARE>(r.o, r.d);
  r.dk = kFilterK * (fabsf(r.d.x) + fabsf(r.d.y) + fabsf(r.d.z));
  return r;
}

// Conservative slab test (intersectUtils.js:2-78).  Accepts whenever the reference's float64
// test could accept: the entry/exit distances carry at most ~4 roundings, and are widened by
// 2^-20 relative before the comparisons.  `entry` returns the widened entry distance.
__device__ __forceinline__ bool box_hit(float x0, float y0, float z0, float x1, float y1, float z1, const RayF& r,
                                        float near_d, float far_d, float& entry) {
  float tx0 = (x0 - r.o.x) * r.inv.x, tx1 = (x1 - r.o.x) * r.inv.x;
  float ty0 = (y0 - r.o.y) * r.inv.y, ty1 = (y1 - r.o.y) * r.inv.y;
  float tz0 = (z0 - r.o.z) * r.inv.z, tz1 = (z1 - r.o.z) * r.inv.z;
  float en = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fminf(tz0, tz1));
  float ex = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fmaxf(tz0, tz1));
  en *= en > 0.0f ? 1.0f - kSlabMargin : 1.0f + kSlabMargin;
  ex *= ex > 0.0f ? 1.0f + kSlabMargin : 1.0f - kSlabMargin;
  entry = en;
  return en <= ex && en <= far_d && ex >= near_d;
}

// ---------------------------------------------------------------------------------------------
// Four-child records: the slab test on centre and half extent.
// ---------------------------------------------------------------------------------------------
// Two float operations in one instruction (sm_100's packed float32 forms; each half rounds as the
// scalar operation does).
struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 f2_make(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_split(f2 a, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {  // a - b as one fused multiply-add by -1
  f2 r;
  const f2 m = f2_make(-1.0f, -1.0f);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(b.v), "l"(m.v), "l"(a.v));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// A ray as the slab test reads it: reciprocal direction, -origin / direction, |reciprocal| and the slack
// of the origin's part.  With inv within 2u of 1 / d, an exact slab bound (p - o) / d of a box with centre c
// and half extent h (before box_centre_half's slack) is a -+ b, a = (c - o) / d and b = h / |d|.  In float32
// t = fma(c, inv, noi) is off by the rounding of noi, which is known exactly (fma(-o, inv, -noi)) and is the
// slack s, and by 3u |a|; r = fma(h, |inv|, s) is at least b + s + 58u b, by the half extent's slack of 64u h.
// |a| <= |a -+ b| + b, so t - r is above the exact entry by at most 5u times the entry's own size, and t + r
// below the exact exit by at most 5u times the exit's.  So entry <= exit (1 + 32u) where the exit is not
// negative, entry <= limit (1 + 32u) and exit >= near (1 - 32u) hold wherever they hold exactly.  All of it is
// relative to distances from the ray's origin, but for s, half an ulp of the origin: slack relative to the
// coordinates made boxes far from the origin overlap (1,000,000 rays on the 80,000-triangle knot moved by 1e6:
// 23.7 ms, now 0.73 ms, and warp-shared 211 and 8.4 ms).
// That takes an o inv that is finite.  For a zero direction component ray_reciprocals sees to it.  (t can be
// infinite still, for a box beside the ray; where the ray is between the box's planes, |c - o| <= h, r is as
// large, and t -+ r a NaN or an infinity that lets the box in.)  Another component whose o inv overflows (a
// direction far from unit length) has an infinite s and rules no box out.  With an infinite o, s is the least
// there is, t infinite, and every box is missed.
struct RaySlab {
  f2 inv, noi, ainv, s;          // x, y
  float invz, noiz, ainvz, sz;
};
__device__ __forceinline__ float slab_slack(float o, float inv, float noi) {
  return fmaxf(fabsf(fmaf(-o, inv, -noi)) * (1.0f + 0x1p-18f), 0x1p-140f);
}
__device__ __forceinline__ RaySlab ray_slab(const RayF& r) {
  RaySlab q;
  const float nx = -r.o.x * r.inv.x, ny = -r.o.y * r.inv.y;
  q.inv = f2_make(r.inv.x, r.inv.y);
  q.noi = f2_make(nx, ny);
  q.ainv = f2_make(fabsf(r.inv.x), fabsf(r.inv.y));
  q.s = f2_make(slab_slack(r.o.x, r.inv.x, nx), slab_slack(r.o.y, r.inv.y, ny));
  q.invz = r.inv.z;
  q.noiz = -r.o.z * r.inv.z;
  q.ainvz = fabsf(r.inv.z);
  q.sz = slab_slack(r.o.z, r.inv.z, q.noiz);
  return q;
}

// The limits of the slab test, widened: a box is entered when entry <= exit, entry <= lim and exit >=
// near.  Every hit has t >= 0, so a negative near acts as 0; with a NaN near nothing is entered.
__device__ __forceinline__ float slab_near(float near_d) { return near_d <= 0.0f ? 0.0f : near_d * (1.0f - 0x1p-19f); }
__device__ __forceinline__ float slab_limit(float lim) { return lim * (1.0f + 0x1p-19f); }
__device__ __forceinline__ float slab_far(float far_d) { return far_d < kInf ? slab_limit(far_d) : kInf; }  // NaN: none

// near and far are distances, and the reference holds them against the ray parameter of its nodes'
// boxes: for a direction that is not of unit length that drops hits by the extent of their leaf's box.
// Parts of leaves, whose boxes the reference does not have, must then not be held against them: a
// direction counts as of unit length while the difference is within the slack of the widened limits.
// Nor against a near that is not a number, which no box of the tree passes but a root that is a leaf does.
// Calls with near <= 0 and no far have nothing to hold (RANGED false).
static inline bool ranged(float near_d, float far_d) { return !(near_d <= 0.0f && far_d >= kInf); }
__device__ __forceinline__ bool free_parts(float3 d, float near_d) {
  return !(fabsf(d.x * d.x + d.y * d.y + d.z * d.z - 1.0f) <= 0x1p-20f) || near_d != near_d;
}

struct ChildBox {
  f2 c, h;
  float cz, hz;
  uint32_t link, part;
};
__device__ __forceinline__ ChildBox load_child(const QuadChild* __restrict__ p) {
  float4 a, b;
  ld8(p, a, b);
  return {f2_make(a.x, a.y), f2_make(a.z, a.w), b.x, b.y, __float_as_uint(b.z), __float_as_uint(b.w)};
}
__device__ __forceinline__ bool child_hit(const ChildBox& c, const RaySlab& r, float near_s, float lim, float& entry) {
  const f2 t = f2_fma(c.c, r.inv, r.noi), q = f2_fma(c.h, r.ainv, r.s);
  const float tz = fmaf(c.cz, r.invz, r.noiz), qz = fmaf(c.hz, r.ainvz, r.sz);
  float nx, ny, fx, fy;
  f2_split(f2_sub(t, q), nx, ny);
  f2_split(f2_add(t, q), fx, fy);
  const float en = max3(nx, ny, tz - qz), ex = min3(fx, fy, tz + qz);
  entry = en;
  return en <= ex * (1.0f + 0x1p-19f) && en <= lim && ex >= near_s;
}

struct Tri {
  float3 a, b, c;
  uint32_t face, flags, material;
};

__device__ __forceinline__ Tri load_tri(const TriRecord* __restrict__ tris, uint32_t k) {
  const TriRecord* t = tris + k;
  float4 p0 = ld4(&t->v[0]), p1 = ld4(&t->v[4]), p2 = ld4(&t->v[8]);
  Tri r;
  r.a = make_float3(p0.x, p0.y, p0.z);
  r.b = make_float3(p0.w, p1.x, p1.y);
  r.c = make_float3(p1.z, p1.w, p2.x);
  r.face = __float_as_uint(p2.y);
  r.flags = __float_as_uint(p2.z);
  r.material = __float_as_uint(p2.w);
  return r;
}

// The side a triangle is tested with: the call's side, or with an array of materials the side of
// the triangle's group material (ThreeRayIntersectUtilities.js:170-205; a material index past the
// array reads as `undefined` and tests like FrontSide).  -1: the triangle is in no group and is
// not tested.
__device__ __forceinline__ int tri_side(const Tri& t, int side, const SideTable& tab) {
  if (!tab.per_material) return side;
  if (t.material == kNoMaterial) return -1;
  return t.material < (uint32_t)tab.n ? (int)tab.side[t.material] : kSideFront;
}

struct Pair {
  float l[6], r[6];
  uint32_t ll, lr, axis, flags;
};

__device__ __forceinline__ Pair load_pair(const PairNode* __restrict__ nodes, uint32_t k) {
  const PairNode* n = nodes + k;
  // two 256-bit loads per record (every pair array is its own allocation of 64-byte records)
  float4 q0, q1, q2, q3;
  ld8(&n->f[0], q0, q1);
  ld8(&n->f[8], q2, q3);
  Pair p;
  p.l[0] = q0.x; p.l[1] = q0.y; p.l[2] = q0.z; p.l[3] = q0.w; p.l[4] = q1.x; p.l[5] = q1.y;
  p.r[0] = q1.z; p.r[1] = q1.w; p.r[2] = q2.x; p.r[3] = q2.y; p.r[4] = q2.z; p.r[5] = q2.w;
  p.ll = __float_as_uint(q3.x);
  p.lr = __float_as_uint(q3.y);
  p.axis = __float_as_uint(q3.z);
  p.flags = __float_as_uint(q3.w);
  return p;
}

// |d| in float-float.
__device__ __forceinline__ ff dir_length(float3 d) {
  ff s = ff_add(ff_add(two_prod(d.x, d.x), two_prod(d.y, d.y)), two_prod(d.z, d.z));
  return ff_sqrt(s);
}

// Full intersection record for a triangle known to be hit, in float-float, rounded once.
// barycoord follows Triangle.getBarycoord: (0, 0, 0) when the triangle's Gram determinant
// |e1 x e2|^2 vanishes at float64 resolution (the reference's `denom === 0` case).
// e = tri_eval_ff of the triangle and ray, tt = its t, dist = the hit's distance.
static __device__ void make_hit(const Tri& t, const RayF& r, const TriFF& e, ff tt, ff dist, bvhc_hit& h) {
  ff3 px = {ff_add(ff_from(r.o.x), ff_mul_f(tt, r.d.x)), ff_add(ff_from(r.o.y), ff_mul_f(tt, r.d.y)),
            ff_add(ff_from(r.o.z), ff_mul_f(tt, r.d.z))};
  h.face_index = t.face;
  h.distance = ff_to_f(dist);
  h.point[0] = ff_to_f(px.x);
  h.point[1] = ff_to_f(px.y);
  h.point[2] = ff_to_f(px.z);
  if (tri_degenerate(t.a, t.b, t.c)) {
    h.barycoord[0] = h.barycoord[1] = h.barycoord[2] = 0.0f;
  } else {
    // W / N, U / N, V / N through one float-float reciprocal (relative error ~2^-44, rounded once
    // to float32)
    const ff rn = ff_div(ff{1.0f, 0.0f}, e.N);
    h.barycoord[0] = ff_to_f(ff_mul(e.W, rn));
    h.barycoord[1] = ff_to_f(ff_mul(e.U, rn));
    h.barycoord[2] = ff_to_f(ff_mul(e.V, rn));
  }
}

__device__ __forceinline__ void store_hit(bvhc_hit* p, const bvhc_hit& h) {
  float4* q = reinterpret_cast<float4*>(p);
  __stcs(q, make_float4(__uint_as_float(h.face_index), h.distance, h.point[0], h.point[1]));
  __stcs(q + 1, make_float4(h.point[2], h.barycoord[0], h.barycoord[1], h.barycoord[2]));
}

__device__ __forceinline__ void store_miss(bvhc_hit* p) {
  float4* q = reinterpret_cast<float4*>(p);
  __stcs(q, make_float4(__uint_as_float(BVHC_NO_HIT), kInf, 0.0f, 0.0f));
  __stcs(q + 1, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
}

// ---------------------------------------------------------------------------------------------
// raycastFirst leaf step shared by both kernel forms.  Candidate hits are ordered with float32 t
// values and their error bounds; float-float only settles candidates the bounds cannot separate
// (the reference keeps the strictly closer one; of exact ties, here, the smaller record, which no order of
// the visits changes.  The form that visits as the reference does, one ray per thread by the direction's
// sign, keeps the one found first, as the reference does).
// ---------------------------------------------------------------------------------------------
constexpr float kTwoU = 1.1920928955078125e-07f;  // 2u

// near <= t |d| <= far from the float32 t and its bound: 1 inside, 0 outside, -1 undecided.
__device__ __forceinline__ int range_filter(float t, float t_err, float dlen, float near_d, float far_d) {
  const float dist = t * dlen;
  const float derr = t_err * dlen + fabsf(dist) * kTwoU + 1e-30f;
  if (dist - derr >= near_d && dist + derr <= far_d) return 1;
  return dist + derr < near_d || dist - derr > far_d ? 0 : -1;
}

// The same and the hit itself in float-float; on a hit, *t is its float-float t.  Out of line, with
// the float-float code in one place: the filters settle nearly every test, and code inlined for the
// rest costs registers in every loop that holds it.
static __device__ __noinline__ bool hit_slow(const TriRecord* __restrict__ tris, uint32_t k, float3 o, float3 d,
                                             int side, float near_d, float far_d, ff* t) {
  const Tri tr = load_tri(tris, k);
  const TriFF e = tri_eval_ff(tr.a, tr.b, tr.c, o, d);
  if (!tri_decide_ff(e, side)) return false;
  *t = tri_t_ff(e);
  const ff dl = ff_mul(*t, dir_length(d));
  return !ff_lt(dl, ff_from(near_d)) && !ff_lt(ff_from(far_d), dl);
}

// Whether the ray hits triangle record k (loaded as `tr`) within [near, far], exactly.
__device__ __forceinline__ bool hit_exact(const MeshDev& m, const Tri& tr, uint32_t k, const RayF& r, float dlen,
                                          int side, float near_d, float far_d) {
  float t, t_err;
  int st = tri_filter(tr.a, tr.b, tr.c, r.o, r.d, r.dk, side, t, t_err);
  if (st > 0) st = range_filter(t, t_err, dlen, near_d, far_d);
  ff tt;
  return st < 0 ? hit_slow(m.tris, k, r.o, r.d, side, near_d, far_d, &tt) : st > 0;
}

struct Best {
  float t, err;
  uint32_t rec;
};

// Offers triangle record k to `best` in float-float: an exact tie goes to the smaller record, or with
// FIRST_FOUND stays with the record found first.
template <bool FIRST_FOUND = false>
static __device__ __noinline__ Best offer_slow(const TriRecord* __restrict__ tris, uint32_t k, float3 o, float3 d,
                                               int side, float near_d, float far_d, Best best) {
  ff tn;
  if (!hit_slow(tris, k, o, d, side, near_d, far_d, &tn)) return best;
  const float err = fabsf(tn.hi) * kTinyRel + 1e-30f;
  bool take = best.rec == 0xFFFFFFFFu || tn.hi + err < best.t - best.err;
  if (!take && !(tn.hi - err > best.t + best.err)) {
    const Tri bt = load_tri(tris, best.rec);
    const ff tb = tri_t_ff(tri_eval_ff(bt.a, bt.b, bt.c, o, d));
    take = ff_lt(tn, tb) || (!FIRST_FOUND && !ff_lt(tb, tn) && k < best.rec);
  }
  return take ? Best{tn.hi, err, k} : best;
}

// Offers triangle record k (loaded as `tr`): the float32 values and bounds decide, else offer_slow.
template <bool FIRST_FOUND = false>
__device__ __forceinline__ void offer_first(const MeshDev& m, const Tri& tr, uint32_t k, const RayF& r, float dlen,
                                            int side, float near_d, float far_d, Best& best) {
  float t, t_err;
  int st = tri_filter(tr.a, tr.b, tr.c, r.o, r.d, r.dk, side, t, t_err);
  if (st > 0) st = range_filter(t, t_err, dlen, near_d, far_d);
  // none yet: best.t is infinite and its bound 0, so every hit is nearer
  if (st > 0) st = t + t_err < best.t - best.err ? 1 : (t - t_err > best.t + best.err ? 0 : -1);
  if (st > 0) best = Best{t, t_err, k};
  else if (st < 0) best = offer_slow<FIRST_FOUND>(m.tris, k, r.o, r.d, side, near_d, far_d, best);
}

template <bool FIRST_FOUND = false>
__device__ __forceinline__ void leaf_first(const MeshDev& m, uint32_t k, const RayF& r, float dlen, int side,
                                           const SideTable& sides, float near_d, float far_d, Best& best) {
  for (;;) {
    const Tri t = load_tri(m.tris, k);
    const int ts = tri_side(t, side, sides);
    if (ts >= 0) offer_first<FIRST_FOUND>(m, t, k, r, dlen, ts, near_d, far_d, best);
    if (t.flags & kTriLast) break;
    ++k;
  }
}

// The same over a run of a four-child record.
__device__ __forceinline__ void run_first(const MeshDev& m, uint32_t link, const RayF& r, float dlen, int side,
                                          const SideTable& sides, float near_d, float far_d, Best& best) {
  const uint32_t first = link & kRunFirst, end = first + ((link >> kRunShift) & 3u) + 1u;
  for (uint32_t k = first; k < end; ++k) {
    const Tri t = load_tri(m.tris, k);
    const int ts = tri_side(t, side, sides);
    if (ts >= 0) offer_first(m, t, k, r, dlen, ts, near_d, far_d, best);
  }
}

// A pending record: the triangle record index in face_index, `t` in distance.  All 32 bytes are
// written, so that the record's DRAM sector is written whole (a half-sector store makes L2 fetch
// the other half first).
__device__ __forceinline__ void store_pending_record(bvhc_hit* o, uint32_t rec, float t) {
  float4* p = reinterpret_cast<float4*>(o);
  __stcs(p, make_float4(__uint_as_float(rec), t, 0.0f, 0.0f));
  __stcs(p + 1, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
}

// A traversal's result left for finalize_first_kernel: a miss record, or pending.
__device__ __forceinline__ void store_first_pending(bvhc_hit* o, const Best& b) {
  if (b.rec == 0xFFFFFFFFu) store_miss(o);
  else store_pending_record(o, b.rec, b.t);
}

// The reported record of the best hit: t, distance, point and barycentrics in float-float.
__device__ __forceinline__ void finish_first(const MeshDev& m, uint32_t rec, const RayF& r, bvhc_hit* o) {
  if (rec == 0xFFFFFFFFu) {
    store_miss(o);
    return;
  }
  Tri t = load_tri(m.tris, rec);
  const TriFF e = tri_eval_ff(t.a, t.b, t.c, r.o, r.d);
  const ff tt = tri_t_ff(e);
  bvhc_hit h;
  make_hit(t, r, e, tt, ff_mul(tt, dir_length(r.d)), h);
  store_hit(o, h);
}

// ---------------------------------------------------------------------------------------------
// raycastFirst (raycastFirst.template.js:19-103, roots loop MeshBVH.js:558-577), one ray per
// thread.  ORDER 0 visits the near child by the sign of the ray direction on the split axis, as
// the reference does; ORDER 1 by the smaller entry distance.  A child whose (widened) entry
// distance is beyond the best hit so far is skipped, which can only drop triangles that are
// farther than that hit.
// ---------------------------------------------------------------------------------------------
template <int ORDER>
__device__ __forceinline__ bool left_first(const Pair& p, const RayF& r, float e0, float e1) {
  if (ORDER == 0) {
    float dir_axis = p.axis == 0 ? r.d.x : (p.axis == 1 ? r.d.y : r.d.z);
    return dir_axis >= 0.0f;
  }
  return e0 <= e1;
}


// Tiled ray order: the ray index space read as rows of `pitch` rays, cut into bands of R = 2^rl
// rows; work item i of a band is the ray at row (i mod 32) / C, column C (i / 32) + i mod C of that
// band with C = 32 / R (pitch a multiple of C), so each warp takes an R x C tile.  For rays
// generated per pixel in row-major order with pitch = the image width, that is an R x C pixel
// block.  Items past the last whole band keep their own index.  A bijection of [0, n): for i below
// the last whole band the row is below R and the column below pitch, so the ray stays in i's band.
__device__ __forceinline__ uint64_t tiled_index(uint64_t i, uint64_t pitch, int rl, uint64_t n) {
  const int cl = 5 - rl;
  const uint64_t band = pitch << rl;
  if (i >= n - n % band) return i;
  const uint64_t b = i / band, r = i - b * band;
  return b * band + ((r & 31u) >> cl) * pitch + ((r >> 5) << cl) + (r & ((1u << cl) - 1u));
}

// Mesh of ray `rid` in a batch: the last mesh whose first ray is <= rid (ray_off is CSR).
__device__ __forceinline__ int mesh_of_ray(const BatchDev& bd, uint64_t rid) {
  int lo = 0, hi = bd.n_meshes - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(bd.ray_off + mid) <= rid) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Pre-pass tiles (classify_kernel, kernels_first.cu).
constexpr int kClsThreads = 256;
constexpr int kClsItems = 8;
constexpr int kClsTile = kClsThreads * kClsItems;  // rays per block
constexpr int kClsWarps = kClsThreads / 32;

}  // namespace dev

static inline unsigned int grid_for(uint64_t n) { return (unsigned int)((n + dev::kBlock - 1) / dev::kBlock); }

// Traversal stack entries a launch may use: 32 when asked for and the tree is shallow enough that
// no traversal pushes more than 31 entries (one per internal level of a root-to-leaf path), else 64.
static inline int stack_entries(const MeshDev& m, int requested) {
  return requested == 32 && m.depth <= 30 ? 32 : 64;
}

// Streaming multiprocessors of the current device.
static inline int sm_count() {
  int dev_id = 0, sms = 0;
  cudaGetDevice(&dev_id);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_id);
  return sms > 0 ? sms : 1;
}

// Whether a view has four-child records, and ones that the phased kernels' stack serves; the entries
// of a group's stack (at most kMaxGroupStack), 0 when the group kernels cannot serve it.  Nothing ever
// overflows either: what a traversal stacks is siblings along one path, and quad_stack counts the most
// siblings of any path.
constexpr int kMaxGroupStack = 96;
static inline bool phased_stack(const MeshDev& m) { return m.quads && m.quad_roots && m.quad_stack <= kMaxStack; }
static inline int group_stack(const MeshDev& m) {
  return m.quads && m.quad_roots && m.quad_stack <= kMaxGroupStack ? (m.quad_stack < 1 ? 1 : m.quad_stack) : 0;
}

// Calls of up to kWideMaxRays rays take the whole warp for each ray, of up to kGroupMaxRays four lanes,
// larger ones one lane.  With few rays the longest ray's chain of dependent steps is the time, and more
// lanes make the chain shorter; with many, the chip is full and the lanes' own work counts.  Rays towards the
// mesh's box, incoherent rays, a camera's, on the 80,000-triangle knot: 4,097 rays 24 us by warps (four lanes: 62,
// one lane 157); 24,000 rays 102, 38, 97 us by warps (four lanes 110, 60, 77); 40,000 rays 158, 53, 148 (127, 70,
// 86); 180,000 rays 227, 104, 176 by fours (one lane 254, 137, 180); 262,145 rays 307, 111, 219 (295, 130, 183).
constexpr uint64_t kWideMaxRays = 24576, kGroupMaxRays = 196608;

// Root-box pre-pass into `queue`, then (single mesh, sort requested) the ray-ordering sort
// (kernels_first.cu).
cudaError_t prepare_queue(const MeshDev& m, const BatchDev* batch, const float* rays, uint64_t n, float near_d,
                          float far_d, bvhc_hit* out, uint32_t* queue, unsigned int* qcount, const RaySort* sort,
                          cudaStream_t stream);

// The root-box pre-pass over a single mesh's rays for the all-hits raycast (kernels_first.cu): rays
// that miss get a hit count of 0 in `miss_counts`, the others are queued in `ids`.
cudaError_t launch_classify_counts(const MeshDev& m, const float* rays, uint64_t n, float near_d, float far_d,
                                   uint32_t* ids, unsigned int* qcount, uint32_t* keys, int kind,
                                   const dev::SceneBox& box, uint32_t* miss_counts, cudaStream_t stream);

}  // namespace bvhc
