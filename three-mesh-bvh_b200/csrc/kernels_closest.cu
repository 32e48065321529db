// closestPointToPoint with minThreshold 0: four lanes per query (the smaller batches take whole warps,
// kernels_wide.cu) over the four-child records, and the 32 queries of a warp through one shared traversal;
// and their launches.
#include <algorithm>
#include <cfloat>

#include "closest.cuh"
#include "group.cuh"

namespace bvhc {
namespace dev {

constexpr int kClosestBlocksPerSm = 8;
constexpr int kClosestRefill = 2 * kGroup;  // idle lanes at which a warp takes new queries

__global__ void __launch_bounds__(kBlock, kClosestBlocksPerSm) closest_point_group_kernel(
    MeshDev m, const float* __restrict__ pts, uint32_t n, float max_t, bvhc_closest* __restrict__ out,
    uint32_t take, int cap) {
  extern __shared__ uint2 s_stack[];
  __shared__ uint2 s_tie[kClosestTies][kBlock];
  const unsigned full = 0xFFFFFFFFu;
  const unsigned lane = threadIdx.x & 31u, j = lane & 3u, base = lane & ~3u;
  const unsigned below = 0x11111111u & ((1u << base) - 1u);  // first lanes of the groups before this one
  uint2* stack = s_stack + (threadIdx.x / kGroup) * (cap + 1);
  const MaxThreshold mx = max_threshold(max_t);
  bool active = false, pending = false, dead = false;  // group-uniform, as in raycast_first_group_kernel
  uint32_t qid = 0, link = 0;
  float3 p = make_float3(0.f, 0.f, 0.f);
  float bound = 0.0f;  // boxes beyond it cannot hold a candidate
  Nearest best = nearest_none();
  int sp = 0, root = 0;
  // this warp's chunks of `take` queries: every (warps of the grid)-th one (no work counter, which calls on
  // different streams would share)
  const uint32_t warps = gridDim.x * (kBlock / 32), chunks = (n + take - 1u) / take;
  uint32_t chunk = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5), pool = 0, pool_end = 0;
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
        store_merged<kGroup>(m.tris, p, best, pending, reinterpret_cast<uint32_t*>(out + qid), s_tie);
        pending = false;
      }
      const unsigned want = __popc(idle) / kGroup;
      if (pool == pool_end && chunk < chunks) {
        pool = chunk * take;
        pool_end = n - pool > take ? pool + take : n;
        chunk += warps;
      }
      const unsigned avail = pool_end - pool, mine = __popc(idle & below);
      if (!active && mine < avail) {
        qid = pool + mine;
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
    if (idle && chunk >= chunks && pool == pool_end) {
      const unsigned walking = __ballot_sync(full, active);
      if (__popc(walking) == kGroup) {  // the last one: all 32 lanes
        if (__ballot_sync(full, pending)) {
          store_merged<kGroup>(m.tris, p, best, pending, reinterpret_cast<uint32_t*>(out + qid), s_tie);
          pending = false;
        }
        const int from = __ffs(walking) - 1;
        if (!active) best = nearest_none();
        qid = __shfl_sync(full, qid, from);
        p.x = __shfl_sync(full, p.x, from);
        p.y = __shfl_sync(full, p.y, from);
        p.z = __shfl_sync(full, p.z, from);
        bound = __shfl_sync(full, bound, from);
        sp = __shfl_sync(full, sp, from);
        link = __shfl_sync(full, link, from);
        dead = __shfl_sync(full, dead, from);
        root = __shfl_sync(full, root, from);
        const int wg = (int)(threadIdx.x >> 5) * kGroups, g = wg + from / kGroup;
        uint2 v[kMaxGroupStack / 32];
        for (int i = 0; i < kMaxGroupStack / 32; ++i)
          if (32 * i + (int)lane < sp) v[i] = s_stack[g * (cap + 1) + 32 * i + lane];
        __syncwarp();
        stack = s_stack + wg * (cap + 1);  // all the groups' stacks
        for (int i = 0; i < kMaxGroupStack / 32; ++i)
          if (32 * i + (int)lane < sp) stack[32 * i + lane] = v[i];
        if (!dead && lane == 0) stack[sp] = make_uint2(link, 0u);
        __syncwarp();
        // eight entries at once while what they add and one depth-first walk fit above the rest
        closest_walk_wide(m, p, mx, stack, kGroups * (cap + 1) - 32 - cap, sp + (dead ? 0 : 1), root, bound, best, s_tie);
        store_merged<32>(m.tris, p, best, true, reinterpret_cast<uint32_t*>(out + qid), s_tie);
        break;
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
          w = box_wanted(c, p, bound, mx, s, l);
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
            if (!beyond(p, t, b.d2 + b.err)) offer_closest(m.tris, p, t, k, candidate(p, t), b, s_tie);
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
                                  bool shared, const uint32_t* queue, uint32_t pitch, int rows_log2,
                                  cudaStream_t stream) {
  if (shared) {
    dev::closest_point_packet_kernel<8><<<grid_for(n), dev::kBlock, 0, stream>>>(m, pts, n, max_t, out, queue, pitch,
                                                                                rows_log2);
    return cudaGetLastError();
  }
  const int cap = group_stack(m);
  if (n <= wide_queries(m)) return launch_closest_wide(m, pts, n, max_t, out, stream);
  const unsigned int resident = (unsigned int)sm_count() * dev::kClosestBlocksPerSm;
  const unsigned int blocks = (n + dev::kBlockGroups - 1) / dev::kBlockGroups;
  // queries a warp takes at once: 100,000 points 503 us by 8 (4: 519, 16: 558, 32: 599), 300,000 the same by all
  const uint32_t take = 8;
  dev::closest_point_group_kernel<<<std::min(blocks, resident), dev::kBlock, group_smem(cap), stream>>>(
      m, pts, n, max_t, out, take, cap);
  return cudaGetLastError();
}

}  // namespace bvhc
