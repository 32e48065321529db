// raycastFirst, one ray per lane in warp-wide phases over the four-child records, persistent; and
// its launch.
#include <algorithm>

#include "traverse.cuh"

namespace bvhc {
namespace dev {

// ---------------------------------------------------------------------------------------------
// raycastFirst for batches that fill the chip.  Every lane holds a ray; a warp alternates between node
// steps (each lane that is at a record tests its four children) and leaf steps (each lane that holds a
// run tests one triangle), whichever more lanes are ready for.  A lane that reaches a leaf keeps it
// pending (up to two) and walks on, so that few lanes stand idle in either step; what it visits before
// the pending triangles have shortened its ray is wasted, and cannot change its nearest hit.  Lanes
// whose rays are finished take new ones from the warp's chunk once kPhasedRefill of them are idle.
//
// What bounds it: instructions issued with part of the lanes (about 18 of 32 in a node step and 16 in
// a leaf step, where descending each lane to its next leaf gave 5.5 in all) and the L1's wavefronts, one
// per lane and load when the lanes are at different records.  1,000,000 rays on the 80,000-triangle
// knot: 1780 us over child pairs, 600 us here (365 instead of 790 warp instructions a ray; two pending
// leaves against none 6%, sorted children against only the nearest first 6%, the stack's first
// twelve entries in shared memory 7%: in thread-local memory lanes at different depths each cost a
// wavefront).
// ---------------------------------------------------------------------------------------------
constexpr int kPhasedBlocksPerSm = 8;     // 64 registers; 7 and 10 blocks within 2% and 10% slower
constexpr unsigned kPhasedChunk = 64;     // rays a warp takes from the work counter at once
constexpr int kPhasedRefill = 12;         // 4 and 24: 5 and 7% slower
constexpr int kPhasedTop = 12;            // stack entries in shared memory (12 KB a block)

template <bool BATCHED, bool MATERIALS, bool RANGED>
__global__ void __launch_bounds__(kBlock, kPhasedBlocksPerSm) raycast_first_phased_kernel(
    MeshDev m, const BatchDev bd, const float* __restrict__ rays, uint32_t n, int side, const SideTable sides,
    float near_d, float far_d, bvhc_hit* __restrict__ out, unsigned long long* __restrict__ work,
    const uint32_t* __restrict__ queue, const unsigned int* __restrict__ qcount) {
  const unsigned full = 0xFFFFFFFFu;
  const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  const uint32_t n_work = queue ? __ldg(qcount) : n;
  const float near_s = slab_near(near_d);
  // a lane's state: `walking` while its traversal goes on (link: a record; or `dead`: its next link is
  // to come off the stack; or a leaf that no pending slot is free for), nl leaves pending (leaf0 being
  // tested, then leaf1); the ray is finished when neither is left
  bool walking = false, dead = false, pending = false;
  int nl = 0;
  uint32_t rid = 0, link = 0, leaf0 = 0, leaf1 = 0;
  RayF r{};
  RaySlab rs{};
  float dlen = 0.0f, lim = 0.0f;
  float lim_hit = 0.0f;  // RANGED: the limit without far
  bool odd = false;      // RANGED
  Best best{kInf, 0.0f, 0xFFFFFFFFu};
  int sp = 0, root = 0, root_end = m.n_roots;
  __shared__ uint2 s_top[kPhasedTop][kBlock];
  uint2 rest[kMaxStack - kPhasedTop];
  auto push = [&](uint32_t l, int key) {
    const uint2 e = make_uint2(l, (uint32_t)key);
    if (sp < kPhasedTop) s_top[sp][threadIdx.x] = e;
    else rest[sp - kPhasedTop] = e;
    ++sp;
  };
  uint32_t pool = 0, pool_end = 0;  // warp-uniform: rays taken and not yet started
  bool drained = false;             // warp-uniform: nothing left to take

  // the newest stacked entry as the next link; `dead` when it is no longer near enough
  auto pop = [&]() {
    dead = true;
    if (sp > 0) {
      --sp;
      const uint2 e = sp < kPhasedTop ? s_top[sp][threadIdx.x] : rest[sp - kPhasedTop];
      link = e.x;
      // (an infinite distance with a child's number in its low bits is no number, and not beyond)
      dead = __uint_as_float(e.y) > (RANGED ? lim_hit : lim);
    } else {
      dead = false;
      walking = ++root < root_end;
      if (walking) link = m.quad_roots[root];
    }
  };

  for (;;) {
    const unsigned idle = __ballot_sync(full, !walking && nl == 0);
    const bool free_lane = (idle >> lane) & 1u;
    if (idle == full || (__popc(idle) >= kPhasedRefill && (!drained || pool < pool_end))) {
      if (free_lane && pending) store_first_pending(out + rid, best);  // finalize_first_kernel completes a hit
      if (free_lane) pending = false;
      const unsigned want = __popc(idle);
      uint32_t avail = pool_end - pool, nb = 0, ne = 0;
      if (want > avail && !drained) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(work, (unsigned long long)kPhasedChunk);
        b = __shfl_sync(full, b, 0);
        drained = b >= n_work;
        if (!drained) {
          nb = (uint32_t)b;
          ne = n_work - nb > kPhasedChunk ? nb + kPhasedChunk : n_work;
        }
      }
      const uint32_t rank = __popc(idle & below);
      if (free_lane && rank < avail + (ne - nb)) {
        rid = rank < avail ? pool + rank : nb + (rank - avail);
        if (queue) rid = __ldg(queue + rid);
        walking = pending = true;
        dead = false;
        r = make_ray(rays, rid);
        rs = ray_slab(r);
        dlen = sqrtf(r.d.x * r.d.x + r.d.y * r.d.y + r.d.z * r.d.z);
        best = Best{kInf, 0.0f, 0xFFFFFFFFu};
        lim = RANGED ? slab_far(far_d) : kInf;
        lim_hit = kInf;
        odd = RANGED && free_parts(r.d, near_d);
        root = 0;
        if (BATCHED) {
          const int mesh = mesh_of_ray(bd, rid);
          root = (int)__ldg(bd.mesh_root_off + mesh);
          root_end = (int)__ldg(bd.mesh_root_off + mesh + 1);
        }
        sp = 0;
        link = m.quad_roots[root];
      }
      if (want <= avail) {
        pool += want;
      } else {
        const uint32_t used = want - avail;
        pool = used < ne - nb ? nb + used : ne;
        pool_end = ne;
      }
      if (!__ballot_sync(full, walking || nl > 0)) {
        if (drained) break;
        continue;
      }
    }
    const int keep = drained && pool == pool_end ? 1 : 33 - kPhasedRefill;
    for (;;) {
      const bool at_node = walking && (dead || !(link & kLeafBit));
      const unsigned nodes = __ballot_sync(full, at_node), leaves = __ballot_sync(full, nl > 0);
      if (__popc(__ballot_sync(full, walking) | leaves) < keep) break;
      if (__popc(nodes) >= __popc(leaves)) {
        if (at_node) {
          bool none = true;
          if (!dead) {
            const QuadNode* q = m.quads + link;
            int key[4];
            uint32_t l[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const ChildBox b = load_child(q->c + c);
              float e;
              const bool free_box = RANGED && odd && b.part;
              const bool h = child_hit(b, rs, free_box ? 0.0f : near_s, free_box ? lim_hit : lim, e);
              key[c] = h ? (int)((__float_as_uint(e) & ~3u) | c) : 0x7FFFFFFF;
              l[c] = b.link;
            }
            auto cas = [&](int a, int b) {
              const int lo = min(key[a], key[b]), hi = max(key[a], key[b]);
              key[a] = lo;
              key[b] = hi;
            };
            cas(0, 1);
            cas(2, 3);
            cas(0, 2);
            cas(1, 3);
            cas(1, 2);
            auto pick = [&](int k) {
              const uint32_t a = (k & 1) ? l[1] : l[0], b = (k & 1) ? l[3] : l[2];
              return (k & 2) ? b : a;
            };
#pragma unroll
            for (int k = 3; k >= 1; --k)
              if (key[k] != 0x7FFFFFFF) push(pick(key[k]), key[k]);
            link = pick(key[0]);
            none = key[0] == 0x7FFFFFFF;
          }
          if (none) pop();
          // a leaf goes to the pending ones and the walk goes on
          if (walking && !dead && (link & kLeafBit) && nl < 2) {
            if (nl == 0) leaf0 = link;
            else leaf1 = link;
            ++nl;
            pop();
          }
        }
      } else {
        if (nl > 0) {
          const uint32_t k = leaf0 & kRunFirst;
          const Tri t = load_tri(m.tris, k);
          const int ts = MATERIALS ? tri_side(t, side, sides) : side;
          if (!MATERIALS || ts >= 0) offer_first(m, t, k, r, dlen, ts, near_d, far_d, best);
          lim_hit = slab_limit((best.t + best.err) * (1.0f + kSlabMargin));
          lim = fminf(lim, lim_hit);
          if (!(leaf0 & ~(kLeafBit | kRunFirst))) {
            leaf0 = leaf1;
            --nl;
            if (walking && !dead && (link & kLeafBit)) {  // the leaf that waited for a slot
              if (nl == 0) leaf0 = link;
              else leaf1 = link;
              ++nl;
              dead = true;
            }
          } else {
            leaf0 += 1u - (1u << kRunShift);  // the next record, one fewer to come
          }
        }
      }
    }
  }
}

}  // namespace dev

cudaError_t launch_raycast_first_phased(const MeshDev& m, const BatchDev* batch, const float* rays, uint64_t n,
                                        int side, const SideTable& sides, float near_d, float far_d, bvhc_hit* out,
                                        unsigned long long* work, cudaStream_t stream, const uint32_t* queue,
                                        const unsigned int* qcount) {
  auto pick = [&](auto k, auto k_ranged) { return dev::ranged(near_d, far_d) ? k_ranged : k; };
  auto kernel =
      batch                ? pick(dev::raycast_first_phased_kernel<true, false, false>, dev::raycast_first_phased_kernel<true, false, true>)
      : sides.per_material ? pick(dev::raycast_first_phased_kernel<false, true, false>, dev::raycast_first_phased_kernel<false, true, true>)
                           : pick(dev::raycast_first_phased_kernel<false, false, false>, dev::raycast_first_phased_kernel<false, false, true>);
  cudaError_t e = cudaMemsetAsync(work, 0, sizeof(unsigned long long), stream);
  if (e != cudaSuccess) return e;
  const BatchDev bd = batch ? *batch : BatchDev{nullptr, nullptr, 0};
  const unsigned int grid = std::min(grid_for(n), (unsigned int)sm_count() * dev::kPhasedBlocksPerSm);
  kernel<<<grid, dev::kBlock, 0, stream>>>(m, bd, rays, (uint32_t)n, side, sides, near_d, far_d, out, work, queue,
                                           qcount);
  return cudaGetLastError();
}

}  // namespace bvhc
