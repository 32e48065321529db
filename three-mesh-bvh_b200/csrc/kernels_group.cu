// raycastFirst in groups of four lanes per ray (group.cuh), persistent; and its launch.
#include <algorithm>

#include "group.cuh"

namespace bvhc {
namespace dev {

// The small batches' kernel: a ray's time is its chain of steps (record load, box tests, choice of the
// next link), and four lanes make the chain of a step short.  4,097 rays on the 10,000-triangle knot:
// 159 us with one lane per ray over child pairs, 50 us here; 80,000 triangles: 157 (one lane over the
// same records) and 64 us.
constexpr int kGroupBlocksPerSm = 8;    // 64 registers; 10 and 12 blocks spill more and measured slower
// Rays a warp takes from the work counter at once: so many warps are resident that with 32 a batch of 40,000 to
// 150,000 rays left a third of them without any (40,000 camera rays 168 us, by 16 111, by 8 86).
constexpr unsigned kGroupChunk = 8;
constexpr int kGroupRefill = 2 * kGroup;  // idle lanes at which a warp takes new rays

template <bool BATCHED, bool MATERIALS, bool RANGED>
__global__ void __launch_bounds__(kBlock, kGroupBlocksPerSm) raycast_first_group_kernel(
    MeshDev m, const BatchDev bd, const float* __restrict__ rays, uint32_t n, int side, const SideTable sides,
    float near_d, float far_d, bvhc_hit* __restrict__ out, unsigned long long* __restrict__ work,
    const uint32_t* __restrict__ queue, const unsigned int* __restrict__ qcount, int cap) {
  extern __shared__ uint2 s_stack[];
  // what only the leaf steps and the ends of a ray need, out of the registers: origin and the filter's
  // factor, direction and its length, ray and end of its roots
  __shared__ float4 s_org[kBlockGroups], s_dir[kBlockGroups];
  __shared__ uint2 s_ray[kBlockGroups];
  const unsigned full = 0xFFFFFFFFu;
  const unsigned lane = threadIdx.x & 31u, j = lane & 3u, base = lane & ~3u;
  const unsigned below = 0x11111111u & ((1u << base) - 1u);  // first lanes of the groups before this one
  uint2* stack = s_stack + (threadIdx.x / kGroup) * (cap + 1);
  const uint32_t n_work = queue ? __ldg(qcount) : n;
  const float near_s = slab_near(near_d);
  bool active = false, pending = false;  // group-uniform: walking a ray; holding a finished one
  bool dead = false;  // group-uniform: at a dead end, no next link found on the stack yet
  const int gi = threadIdx.x / kGroup;
  RaySlab rg{};
  float lim = 0.0f, lim_hit = 0.0f;    // lim_hit (RANGED): without far
  bool odd = false;                    // RANGED
  Best best{kInf, 0.0f, 0xFFFFFFFFu};  // this lane's nearest hit
  uint32_t link = 0;
  int sp = 0, root = 0;
  auto load_ray = [&](RayF& r) {
    const float4 o = s_org[gi];
    r.o = make_float3(o.x, o.y, o.z);
    r.dk = o.w;
    const float4 d = s_dir[gi];
    r.d = make_float3(d.x, d.y, d.z);
    return d.w;
  };
  uint32_t pool = 0, pool_end = 0;  // warp-uniform: rays taken and not yet started
  bool drained = false;             // warp-uniform: nothing left to take
  if (!work) {                      // one ray per group of the grid
    pool = (blockIdx.x * kBlock + (threadIdx.x & ~31u)) / kGroup;
    pool_end = pool + kGroups < n_work ? pool + kGroups : n_work;
    if (pool > pool_end) pool = pool_end;
    drained = true;
  }

  // the stack is empty: on to the next root, or the ray is finished
  auto next_root = [&]() {
    sp = 0;
    dead = false;
    if (++root < (int)s_ray[gi].y) {
      link = m.quad_roots[root];
    } else {
      active = false;
      pending = true;
    }
  };

  for (;;) {
    const unsigned idle = __ballot_sync(full, !active);
    if (idle == full || (__popc(idle) >= kGroupRefill && (!drained || pool < pool_end))) {
      // the finished rays' four candidates to one, and its pending record
      if (__ballot_sync(full, pending)) {
#pragma unroll
        for (int x = 1; x <= 2; x <<= 1) {
          Best o;
          o.t = __shfl_xor_sync(full, best.t, x);
          o.err = __shfl_xor_sync(full, best.err, x);
          o.rec = __shfl_xor_sync(full, best.rec, x);
          if (!pending || o.rec == 0xFFFFFFFFu || o.t - o.err > best.t + best.err) continue;
          if (o.t + o.err < best.t - best.err) {
            best = o;
          } else {  // both are hits: the side, near and far of the call hold for them
            RayF r;
            load_ray(r);
            best = offer_slow(m.tris, o.rec, r.o, r.d, kSideDouble, 0.0f, kInf, best);
          }
        }
        if (pending && j == 0) store_first_pending(out + s_ray[gi].x, best);  // finalize_first_kernel completes a hit
        pending = false;
      }
      const unsigned want = __popc(idle) / kGroup;
      if (pool == pool_end && !drained) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(work, (unsigned long long)kGroupChunk);
        b = __shfl_sync(full, b, 0);
        drained = b >= n_work;
        if (!drained) {
          pool = (uint32_t)b;
          pool_end = n_work - pool > kGroupChunk ? pool + kGroupChunk : n_work;
        }
      }
      const unsigned avail = pool_end - pool;
      const unsigned mine = __popc(idle & below);
      if (!active && mine < avail) {
        uint32_t rid = pool + mine;
        if (queue) rid = __ldg(queue + rid);
        active = true;
        const RayF r = make_ray(rays, rid);
        rg = ray_slab(r);
        best = Best{kInf, 0.0f, 0xFFFFFFFFu};
        lim = RANGED ? slab_far(far_d) : kInf;
        lim_hit = kInf;
        odd = RANGED && free_parts(r.d, near_d);
        int root_end = m.n_roots;
        root = 0;
        if (BATCHED) {
          int mesh = mesh_of_ray(bd, rid);
          root = (int)__ldg(bd.mesh_root_off + mesh);
          root_end = (int)__ldg(bd.mesh_root_off + mesh + 1);
        }
        sp = 0;
        link = m.quad_roots[root];
        if (j == 0) {
          s_dir[gi] = make_float4(r.d.x, r.d.y, r.d.z, sqrtf(r.d.x * r.d.x + r.d.y * r.d.y + r.d.z * r.d.z));
          s_org[gi] = make_float4(r.o.x, r.o.y, r.o.z, r.dk);
          s_ray[gi] = make_uint2((uint32_t)rid, (uint32_t)root_end);
        }
      }
      __syncwarp();
      pool += want < avail ? want : avail;
      if (!__ballot_sync(full, active)) {
        if (drained) break;
        continue;
      }
    }
    // node steps, while no more groups wait at leaves than are at records
    bool at_node = active && (dead || !(link & kLeafBit));
    unsigned nodes = __ballot_sync(full, at_node), leaves = __ballot_sync(full, active) & ~nodes;
    while (nodes && __popc(nodes) >= __popc(leaves)) {
      bool h = false, ok = false;
      float e = 0.0f;
      uint32_t l = 0u;
      uint2 top = make_uint2(0u, 0u);
      if (at_node) {
        if (sp > (int)j) {
          top = stack[sp - 1 - (int)j];
          ok = __uint_as_float(top.y) <= (RANGED ? lim_hit : lim);
        }
        if (!dead) {
          const ChildBox c = load_child(m.quads[link].c + j);
          const bool free_box = RANGED && odd && c.part;
          h = child_hit(c, rg, free_box ? 0.0f : near_s, free_box ? lim_hit : lim, e);
          l = c.link;
        }
      }
      const unsigned hits = (__ballot_sync(full, h) >> base) & 0xFu, oks = (__ballot_sync(full, ok) >> base) & 0xFu;
      int rank;
      unsigned first;
      group_rank(h ? (int)((__float_as_uint(e) & ~3u) | j) : 0x7FFFFFFF, rank, first);
      // The nearest child is next and the others are stacked, farthest first (within `cap`: what is
      // stacked is siblings along one path, which the host counted).  At a dead end the newest of the
      // top four entries that is still nearer than the best hit is next.
      const unsigned pop = (unsigned)__ffs(oks) - 1u;
      const uint32_t next = __shfl_sync(full, hits ? l : top.x, base + (hits ? first : pop & 3u));
      if (at_node) {
        const int nh = __popc(hits);
        if (h && rank) stack[sp + nh - 1 - rank] = make_uint2(l, __float_as_uint(e));
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
    // leaf step: four triangles of each group that holds a leaf
    const bool at_leaf = active && !dead && (link & kLeafBit);
    if (at_leaf && j <= ((link >> kRunShift) & 3u)) {
      const uint32_t k = (link & kRunFirst) + j;
      const Tri t = load_tri(m.tris, k);
      const int ts = MATERIALS ? tri_side(t, side, sides) : side;
      RayF r;
      const float dlen = load_ray(r);
      if (!MATERIALS || ts >= 0) offer_first(m, t, k, r, dlen, ts, near_d, far_d, best);
    }
    const float nl = slab_limit(group_min((best.t + best.err) * (1.0f + kSlabMargin)));
    bool ok = false;
    uint2 top = make_uint2(0u, 0u);
    if (at_leaf) {
      lim = fminf(lim, nl);
      if (RANGED) lim_hit = fminf(lim_hit, nl);
      if (sp > (int)j) {
        top = stack[sp - 1 - (int)j];
        ok = __uint_as_float(top.y) <= (RANGED ? lim_hit : lim);
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

}  // namespace dev

cudaError_t launch_raycast_first_group(const MeshDev& m, const BatchDev* batch, const float* rays, uint64_t n, int side,
                                       const SideTable& sides, float near_d, float far_d, bvhc_hit* out,
                                       unsigned long long* work, cudaStream_t stream, const uint32_t* queue,
                                       const unsigned int* qcount) {
  const int cap = group_stack(m);
  const size_t smem = group_smem(cap);
  auto pick = [&](auto k, auto k_ranged) { return dev::ranged(near_d, far_d) ? k_ranged : k; };
  auto kernel =
      batch                ? pick(dev::raycast_first_group_kernel<true, false, false>, dev::raycast_first_group_kernel<true, false, true>)
      : sides.per_material ? pick(dev::raycast_first_group_kernel<false, true, false>, dev::raycast_first_group_kernel<false, true, true>)
                           : pick(dev::raycast_first_group_kernel<false, false, false>, dev::raycast_first_group_kernel<false, false, true>);
  const uint64_t resident = (uint64_t)sm_count() * dev::kGroupBlocksPerSm;
  const uint64_t blocks = (n + dev::kBlockGroups - 1) / dev::kBlockGroups;
  // one ray per group where the grid holds that many: no work counter to reset and to draw from
  const bool fits = blocks <= resident;
  if (!fits) {
    cudaError_t e = cudaMemsetAsync(work, 0, sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return e;
  }
  const BatchDev bd = batch ? *batch : BatchDev{nullptr, nullptr, 0};
  kernel<<<(unsigned int)std::min(blocks, resident), dev::kBlock, smem, stream>>>(
      m, bd, rays, (uint32_t)n, side, sides, near_d, far_d, out, fits ? nullptr : work, queue, qcount, cap);
  return cudaGetLastError();
}

}  // namespace bvhc
