// closestPointToPoint with minThreshold 0: four lanes per query over the four-child records, and the 32
// queries of a warp through one shared traversal; and their launches.
#include <algorithm>
#include <cfloat>

#include "closest.cuh"
#include "group.cuh"

namespace bvhc {
namespace dev {

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
  const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
  const float e43 = d4 - d3, e56 = d5 - d6;
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

// Whether candidate `cand` beats `b` where their float32 distances do not tell: the same vertex is an
// exact tie, else the float-float distances decide; an exact tie goes to the smaller faceIndex.
static __device__ __noinline__ bool closer_slow(const TriRecord* __restrict__ tris, float3 p, uint32_t cand,
                                                uint32_t b) {
  const Tri t = load_tri(tris, cand & kRunFirst), u = load_tri(tris, b & kRunFirst);
  const uint32_t tv = cand >> kRunShift, uv = b >> kRunShift;
  if (tv != 3u && uv != 3u && same_vertex(t, tv, u, uv)) return t.face < u.face;
  const ff d = closest_ff(p, t.a, t.b, t.c).d2, e = closest_ff(p, u.a, u.b, u.c).d2;
  return ff_lt(d, e) || (!ff_lt(e, d) && t.face < u.face);
}

// Offers triangle t (record k) at candidate c to a lane's best.  Candidates are ranked by exact distance,
// then by faceIndex, a total order that does not depend on the order of the offers.  What float32 and
// the shared vertex do not settle is kept beside the best one for the finalize kernel: most of it is
// overtaken by a nearer triangle later in the walk, and float-float code in the loop is fetched and
// executed by whole warps for one lane.
__device__ __forceinline__ void offer_closest(const TriRecord* __restrict__ tris, float3 p, const Tri& t, uint32_t k,
                                              const Candidate& c, Nearest& b, uint2 (*s_tie)[kBlock]) {
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

constexpr int kClosestBlocksPerSm = 8;
constexpr int kClosestRefill = 2 * kGroup;  // idle lanes at which a warp takes new queries

template <bool MAXED>
__global__ void __launch_bounds__(kBlock, kClosestBlocksPerSm) closest_point_group_kernel(
    MeshDev m, const float* __restrict__ pts, uint32_t n, float max_t, bvhc_closest* __restrict__ out,
    const uint32_t* __restrict__ queue, uint32_t pitch, int rows_log2, int cap) {
  extern __shared__ uint2 s_stack[];
  __shared__ uint2 s_tie[kClosestTies][kBlock];
  const unsigned full = 0xFFFFFFFFu;
  const unsigned lane = threadIdx.x & 31u, j = lane & 3u, base = lane & ~3u;
  const unsigned below = 0x11111111u & ((1u << base) - 1u);  // first lanes of the groups before this one
  uint2* stack = s_stack + (threadIdx.x / kGroup) * (cap + 1);
  const ff max2 = two_prod(max_t, max_t);
  // box distances outside [max_lo, max_hi) are decided by their float32 value (see under_max)
  const float max_lo = max2.hi * (1.0f - kSlabMargin) * (1.0f - 0x1p-19f), max_hi = max2.hi * (1.0f + 0x1p-18f);
  bool active = false, pending = false, dead = false;  // group-uniform, as in raycast_first_group_kernel
  uint32_t qid = 0, link = 0;
  float3 p = make_float3(0.f, 0.f, 0.f);
  float bound = 0.0f;  // boxes beyond it cannot hold a candidate
  Nearest best = nearest_none();
  int sp = 0, root = 0;
  // this warp's chunks of 32 queries: every (warps of the grid)-th one
  const uint32_t warps = gridDim.x * (kBlock / 32), chunks = (n + 31u) / 32u;
  uint32_t chunk = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5), pool = 0, pool_end = 0;
  if (chunks <= warps / 4) {  // few queries: eight, one per group, for each warp
    pool = min(chunk * kGroups, n);
    pool_end = min(pool + kGroups, n);
    chunk = chunks;
  }
  auto next_root = [&]() {
    sp = 0;
    dead = false;
    if (++root < m.n_roots) {
      link = m.quad_roots[root];
    } else {
      active = false;
      pending = true;
    }
  };
  for (;;) {
    const unsigned idle = __ballot_sync(full, !active);
    if (idle == full || (__popc(idle) >= kClosestRefill && (chunk < chunks || pool < pool_end))) {
      if (__ballot_sync(full, pending)) {
        // the four lanes' candidates to one and what is not settled against it
        const int key = best.rec == kNoRecord ? 0x7FFFFFFF : (int)((__float_as_uint(best.d2) & ~3u) | j);
        int rank;
        unsigned first;
        group_rank(key, rank, first);
        const unsigned src = base + first;
        const float hi = __shfl_sync(full, best.d2 + best.err, src);
        uint32_t rec = __shfl_sync(full, best.rec, src);
        const uint32_t face = __shfl_sync(full, best.face, src);
        const float qx = __shfl_sync(full, best.q.x, src), qy = __shfl_sync(full, best.q.y, src),
                    qz = __shfl_sync(full, best.q.z, src);
        bool extra = lane != src && best.rec != kNoRecord && !(best.d2 - best.err > hi);
        const bool same = extra && (rec >> kRunShift) != 3u && (best.rec >> kRunShift) != 3u && best.q.x == qx &&
                          best.q.y == qy && best.q.z == qz;
        extra = extra && !same;
        // of the lanes at the same vertex the smallest faceIndex
        uint32_t f = same || lane == src ? best.face : 0xFFFFFFFFu;
        f = min(f, __shfl_xor_sync(full, f, 1));
        f = min(f, __shfl_xor_sync(full, f, 2));
        const unsigned winner = (__ballot_sync(full, (same || lane == src) && best.face == f) >> base) & 0xFu;
        rec = __shfl_sync(full, best.rec, base + (f != face && winner ? (unsigned)__ffs(winner) - 1u : first));
        int mine = extra ? 1 : 0;
        for (int k = 0; k < best.ties; ++k) mine += !(__uint_as_float(s_tie[k][threadIdx.x].y) > hi);
        if (!pending || best.rec == kNoRecord) mine = 0;
        const int a1 = __shfl_xor_sync(full, mine, 1), pair = mine + a1, other = __shfl_xor_sync(full, pair, 2);
        const int total = pair + other;
        int at = ((j & 1u) ? a1 : 0) + ((j & 2u) ? other : 0);
        if (__ballot_sync(full, pending && total > kClosestTies)) {
          // more than the record holds: settled here
          const bool over = pending && total > kClosestTies;
          uint32_t mine_rec = best.rec;
          if (over && mine_rec != kNoRecord)
            for (int k = 0; k < best.ties; ++k)
              if (closer_slow(m.tris, p, s_tie[k][threadIdx.x].x, mine_rec)) mine_rec = s_tie[k][threadIdx.x].x;
#pragma unroll
          for (int x = 1; x <= 2; x <<= 1) {
            const uint32_t o = __shfl_xor_sync(full, mine_rec, x);
            if (over && o != kNoRecord && (mine_rec == kNoRecord || closer_slow(m.tris, p, o, mine_rec))) mine_rec = o;
          }
          if (over) {
            rec = mine_rec;
            mine = 0;
          }
        }
        if (pending) {  // closest_point_finalize_kernel completes it
          uint32_t* o = reinterpret_cast<uint32_t*>(out + qid);
          if (j == 0) {
            o[0] = rec;
            o[1] = total > kClosestTies ? 0u : (uint32_t)total;
          }
          if (mine) {
            if (extra) o[2 + at++] = best.rec;
            for (int k = 0; k < best.ties; ++k)
              if (!(__uint_as_float(s_tie[k][threadIdx.x].y) > hi)) o[2 + at++] = s_tie[k][threadIdx.x].x;
          }
        }
        pending = false;
      }
      const unsigned want = __popc(idle) / kGroup;
      if (pool == pool_end && chunk < chunks) {
        pool = chunk * 32u;
        pool_end = n - pool > 32u ? pool + 32u : n;
        chunk += warps;
      }
      const unsigned avail = pool_end - pool, mine = __popc(idle & below);
      if (!active && mine < avail) {
        qid = pool + mine;
        if (queue) qid = __ldg(queue + qid);
        else if (pitch) qid = (uint32_t)tiled_index(qid, pitch, rows_log2, n);
        const float* q = pts + 3 * (size_t)qid;
        p = make_float3(__ldg(q), __ldg(q + 1), __ldg(q + 2));
        // a point that is not finite reaches no leaf
        active = fabsf(p.x) <= FLT_MAX && fabsf(p.y) <= FLT_MAX && fabsf(p.z) <= FLT_MAX;
        pending = !active;
        best = nearest_none();
        bound = FLT_MAX;
        dead = false;
        root = 0;
        sp = 0;
        link = m.quad_roots[0];
      }
      pool += want < avail ? want : avail;
      if (!__ballot_sync(full, active)) {
        if (chunk >= chunks && pool == pool_end && !__ballot_sync(full, pending)) break;
        continue;
      }
    }
    // node steps, while no more groups wait at leaves than are at records
    bool at_node = active && (dead || !(link & kLeafBit));
    unsigned nodes = __ballot_sync(full, at_node), leaves = __ballot_sync(full, active) & ~nodes;
    while (nodes && __popc(nodes) >= __popc(leaves)) {
      bool w = false, ok = false;
      float s = 0.0f;
      uint32_t l = 0u;
      uint2 top = make_uint2(0u, 0u);
      if (at_node) {
        if (sp > (int)j) {
          top = stack[sp - 1 - (int)j];
          ok = __uint_as_float(top.y) <= bound;
        }
        if (!dead) {
          const BoxChild* c = m.boxes[link].c + j;
          float4 a, b;
          ld8(c, a, b);
          l = __float_as_uint(b.z);
          const float dx = max3(a.x - p.x, p.x - a.w, 0.0f), dy = max3(a.y - p.y, p.y - b.x, 0.0f),
                      dz = max3(a.z - p.z, p.z - b.y, 0.0f);
          s = dx * dx + dy * dy + dz * dz;
          w = s <= bound;
          if (MAXED && w && !(s < max_lo) && __float_as_uint(b.w) == 0u) w = s < max_hi && under_max_slow(c, p, max2);
        }
      }
      const unsigned hits = (__ballot_sync(full, w) >> base) & 0xFu, oks = (__ballot_sync(full, ok) >> base) & 0xFu;
      int rank;
      unsigned first;
      group_rank(w ? (int)((__float_as_uint(s) & ~3u) | j) : 0x7FFFFFFF, rank, first);
      const unsigned pop = (unsigned)__ffs(oks) - 1u;
      const uint32_t next = __shfl_sync(full, hits ? l : top.x, base + (hits ? first : pop & 3u));
      if (at_node) {
        const int nh = __popc(hits);
        if (w && rank) stack[sp + nh - 1 - rank] = make_uint2(l, __float_as_uint(s));
        link = next;
        sp += hits ? nh - 1 : (oks ? -(int)(pop + 1u) : -kGroup);
        dead = !hits && !oks;
        if (dead && sp <= 0) next_root();
      }
      __syncwarp();
      at_node = active && (dead || !(link & kLeafBit));
      nodes = __ballot_sync(full, at_node);
      leaves = __ballot_sync(full, active) & ~nodes;
    }
    if (!leaves) continue;
    // leaf step: up to four triangles of each group that holds a run
    const bool at_leaf = active && !dead && (link & kLeafBit);
    if (at_leaf && j <= ((link >> kRunShift) & 3u)) {
      const uint32_t k = (link & kRunFirst) + j;
      const Tri t = load_tri(m.tris, k);
      offer_closest(m.tris, p, t, k, candidate(p, t), best, s_tie);
    }
    const float nb = group_min(fminf((best.d2 + best.err) * (1.0f + 0x1p-18f), FLT_MAX));
    bool ok = false;
    uint2 top = make_uint2(0u, 0u);
    if (at_leaf) {
      bound = nb;
      if (sp > (int)j) {
        top = stack[sp - 1 - (int)j];
        ok = __uint_as_float(top.y) <= bound;
      }
    }
    const unsigned oks = (__ballot_sync(full, ok) >> base) & 0xFu;
    const unsigned pop = (unsigned)__ffs(oks) - 1u;
    const uint32_t next = __shfl_sync(full, top.x, base + (pop & 3u));
    if (at_leaf) {
      link = next;
      sp -= oks ? (int)(pop + 1u) : kGroup;
      dead = !oks;
      if (dead && sp <= 0) next_root();
    }
    __syncwarp();
  }
}

// Squared distance from p to the box's centre: the visiting order's tie-break when both child
// boxes hold p (both scores 0), which the scores alone cannot order.
__device__ __forceinline__ float centre_d2(const float* b, float3 p) {
  const float dx = 0.5f * (b[0] + b[3]) - p.x, dy = 0.5f * (b[1] + b[4]) - p.y, dz = 0.5f * (b[2] + b[5]) - p.z;
  return dx * dx + dy * dy + dz * dz;
}

// Whether the right child should be visited first: the smaller score, equal scores by the nearer
// centre (the warp-cooperative forms; the per-query kernel keeps the reference's order).  The
// centre distances are computed only on equal scores (written as a branch: as one expression they
// were evaluated on every node, 4% of the grid's time).
__device__ __forceinline__ bool right_nearer(const Pair& pr, float s0, float s1, float3 p) {
  if (s1 != s0) return s1 < s0;
  return centre_d2(pr.r, p) < centre_d2(pr.l, p);
}

// Whether the triangle's box is farther than the best candidate for certain: at most 4 roundings above
// the exact value's relative 2^-22, so the 2^-20 shrink keeps the distance a lower bound.
__device__ __forceinline__ bool beyond(float3 p, const Tri& t, const Nearest& b) {
  const float dx = fmaxf(fmaxf(fminf(t.a.x, fminf(t.b.x, t.c.x)) - p.x, p.x - fmaxf(t.a.x, fmaxf(t.b.x, t.c.x))), 0.0f);
  const float dy = fmaxf(fmaxf(fminf(t.a.y, fminf(t.b.y, t.c.y)) - p.y, p.y - fmaxf(t.a.y, fmaxf(t.b.y, t.c.y))), 0.0f);
  const float dz = fmaxf(fmaxf(fminf(t.a.z, fminf(t.b.z, t.c.z)) - p.z, p.z - fmaxf(t.a.z, fmaxf(t.b.z, t.c.z))), 0.0f);
  return (dx * dx + dy * dy + dz * dz) * (1.0f - 0x1p-20f) > b.d2 + b.err;
}

// ---------------------------------------------------------------------------------------------
// closestPointToPoint, warp-cooperative form for spatially coherent queries (grids, SDF samples)
// with minThreshold 0.  The 32 queries of a warp walk the tree together with one shared stack of
// links: a child is entered when any lane wants it (its score under maxThreshold^2, decided
// exactly, and not certainly above that lane's best), and each lane keeps, for the current node
// and for every stacked child, whether it wants it (its own score, or NaN for "no").  A lane only
// tests the triangles of leaves it wants, so every lane reaches exactly the leaves its own
// traversal would and its result is the minimum over the same candidates: which leaves a query
// reaches, and so the "null iff no leaf is reached" rule, does not depend on the visiting order,
// and leaves skipped because of the best distance cannot hold a strictly closer triangle.  (With
// minThreshold > 0 the reference stops at the first triangle below it in its own order, which a
// shared order would not reproduce; those calls use the per-query kernel.)
// ---------------------------------------------------------------------------------------------
template <int MINB>
__global__ void __launch_bounds__(kBlock, MINB) closest_point_packet_kernel(
    MeshDev m, const float* __restrict__ pts, uint64_t n, float max_t, bvhc_closest* __restrict__ out,
    const uint32_t* __restrict__ queue, uint64_t pitch, int rows_log2) {
  __shared__ uint32_t s_link[kWarps][kMaxStack];
  __shared__ uint2 s_tie[kClosestTies][kBlock];
  const int w = threadIdx.x >> 5;
  const unsigned full = 0xFFFFFFFFu, lane = threadIdx.x & 31u;
  const uint64_t n_work = n;
  if ((uint64_t)blockIdx.x * blockDim.x >= n_work) return;  // block-uniform
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < n_work;
  if (valid && queue) i = __ldg(queue + i);
  else if (valid && pitch) i = tiled_index(i, pitch, rows_log2, n);  // tiles of grid points
  float3 p = make_float3(0.f, 0.f, 0.f);
  if (valid) p = make_float3(__ldg(pts + 3 * i), __ldg(pts + 3 * i + 1), __ldg(pts + 3 * i + 2));
  const ff max2 = two_prod(max_t, max_t);
  const float kNo = __int_as_float(0x7FFFFFFF);  // NaN: "this lane does not want the entry"
  Nearest b = nearest_none();
  float lane_s[kMaxStack];
  bool overflow = false;
  for (int root = 0; root < m.n_roots && !overflow; ++root) {
    uint32_t link = m.roots[root];
    bool act = valid;  // this lane wants the current node (a root leaf has no bounds test)
    int sp = 0;
    for (;;) {
      bool pop = false;
      if (link & kLeafBit) {
        if (link != kEmptyLeaf && act) {
          uint32_t k = link & ~kLeafBit;
          for (;;) {
            Tri t = load_tri(m.tris, k);
            if (!beyond(p, t, b)) offer_closest(m.tris, p, t, k, candidate(p, t), b, s_tie);
            if (t.flags & kTriLast) break;
            ++k;
          }
        }
        pop = true;
      } else {
        Pair pr = load_pair(m.nodes, link);
        float s0 = box_score(pr.l, p), s1 = box_score(pr.r, p);
        float best_hi = b.d2 + b.err;
        bool w0 = act && s0 * (1.0f - kSlabMargin) <= best_hi && under_max(s0, pr.l, p, max2);
        bool w1 = act && s1 * (1.0f - kSlabMargin) <= best_hi && under_max(s1, pr.r, p, max2);
        unsigned b0 = __ballot_sync(full, w0), b1 = __ballot_sync(full, w1);
        if (b0 && b1) {
          // nearer child first by majority of the lanes that want both (a lane wanting one prefers it)
          bool pref_right = (w0 && w1) ? right_nearer(pr, s0, s1, p) : w1;
          unsigned voters = __ballot_sync(full, w0 || w1);
          bool right_first = 2 * __popc(__ballot_sync(full, (w0 || w1) && pref_right)) > __popc(voters);
          if (sp >= kMaxStack) {
            if (lane == 0) atomicOr(m.err, kErrStackOverflow);
            b = nearest_none();
            overflow = true;
            break;
          }
          if (lane == 0) s_link[w][sp] = right_first ? pr.ll : pr.lr;
          lane_s[sp] = right_first ? (w0 ? s0 : kNo) : (w1 ? s1 : kNo);
          ++sp;
          link = right_first ? pr.lr : pr.ll;
          act = right_first ? w1 : w0;
          __syncwarp();
        } else if (b0) {
          link = pr.ll;
          act = w0;
        } else if (b1) {
          link = pr.lr;
          act = w1;
        } else {
          pop = true;
        }
      }
      if (pop) {
        bool found = false;
        while (sp > 0) {
          --sp;
          bool ok = lane_s[sp] * (1.0f - kSlabMargin) <= b.d2 + b.err;  // false for NaN
          if (__ballot_sync(full, ok)) {
            link = s_link[w][sp];
            act = ok;
            found = true;
            break;
          }
        }
        if (!found) break;
      }
    }
  }
  if (valid) {  // closest_point_finalize_kernel completes it
    uint32_t* o = reinterpret_cast<uint32_t*>(out + i);
    o[0] = b.rec;
    o[1] = (uint32_t)b.ties;
    for (int k = 0; k < b.ties; ++k) o[2 + k] = s_tie[k][threadIdx.x].x;
  }
}


}  // namespace dev

cudaError_t launch_closest_phased(const MeshDev& m, const float* pts, uint32_t n, float max_t, bvhc_closest* out,
                                  const uint32_t* queue, uint32_t pitch, int rows_log2, cudaStream_t stream) {
  if (pitch || queue) {
    dev::closest_point_packet_kernel<8><<<grid_for(n), dev::kBlock, 0, stream>>>(m, pts, n, max_t, out, queue, pitch,
                                                                                rows_log2);
    return cudaGetLastError();
  }
  const int cap = group_stack(m);
  const bool maxed = !(max_t >= dev::kInf);
  auto kernel = maxed ? dev::closest_point_group_kernel<true> : dev::closest_point_group_kernel<false>;
  const unsigned int resident = (unsigned int)sm_count() * dev::kClosestBlocksPerSm;
  const unsigned int blocks = (n + dev::kBlockGroups - 1) / dev::kBlockGroups;
  kernel<<<std::min(blocks, resident), dev::kBlock, group_smem(cap), stream>>>(m, pts, n, max_t, out, queue, pitch,
                                                                              rows_log2, cap);
  return cudaGetLastError();
}

}  // namespace bvhc
