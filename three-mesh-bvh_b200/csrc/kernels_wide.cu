// The whole warp on one query: raycastFirst and closestPointToPoint for the smaller batches; and their
// launches.
#include <algorithm>
#include <cfloat>

#include "closest.cuh"
#include "group.cuh"

namespace bvhc {
namespace dev {

template <bool MATERIALS>
__global__ void __launch_bounds__(kBlock) raycast_first_wide_kernel(MeshDev m, const BatchDev bd, bool batched,
                                                                    const float* __restrict__ rays, uint32_t n, int side,
                                                                    const SideTable sides, float near_d, float far_d,
                                                                    bool ranged_call, bvhc_hit* __restrict__ out,
                                                                    const uint32_t* __restrict__ queue,
                                                                    const unsigned int* __restrict__ qcount, int cap) {
  extern __shared__ uint2 s_stack[];
  const unsigned full = 0xFFFFFFFFu, lane = threadIdx.x & 31u, j = lane & 3u;
  uint2* stack = s_stack + (threadIdx.x >> 5) * cap;
  const uint32_t n_work = queue ? __ldg(qcount) : n;
  const float near_s = slab_near(near_d);
  for (uint32_t w = blockIdx.x * kWarps + (threadIdx.x >> 5); w < n_work; w += gridDim.x * kWarps) {
    const uint32_t rid = queue ? __ldg(queue + w) : w;
    const RayF r = make_ray(rays, rid);
    const RaySlab rs = ray_slab(r);
    const float dlen = sqrtf(r.d.x * r.d.x + r.d.y * r.d.y + r.d.z * r.d.z);
    const bool odd = ranged_call && free_parts(r.d, near_d);
    int root = 0, root_end = m.n_roots;
    if (batched) {
      const int mesh = mesh_of_ray(bd, rid);
      root = (int)__ldg(bd.mesh_root_off + mesh);
      root_end = (int)__ldg(bd.mesh_root_off + mesh + 1);
    }
    Best best{kInf, 0.0f, 0xFFFFFFFFu};
    float lim = slab_far(far_d), lim_hit = kInf;
    for (; root < root_end; ++root) {
      int sp = 1;
      if (lane == 0) stack[0] = make_uint2(m.quad_roots[root], __float_as_uint(-kInf));
      __syncwarp();
      while (sp > 0) {
        WideEntry e = wide_take(stack, sp, lane);
        e.on = e.on && e.key <= lim_hit;
        const bool leaf = e.on && (e.link & kLeafBit);
        bool enter = false;
        uint32_t link = 0u;
        float key = 0.0f;
        if (e.on && !leaf) {
          const ChildBox c = load_child(m.quads[e.link].c + j);
          const bool free_box = odd && c.part;
          enter = child_hit(c, rs, free_box ? 0.0f : near_s, free_box ? lim_hit : lim, key);
          link = c.link;
        }
        if (leaf && j <= ((e.link >> kRunShift) & 3u)) {
          const uint32_t k = (e.link & kRunFirst) + j;
          const Tri t = load_tri(m.tris, k);
          const int ts = MATERIALS ? tri_side(t, side, sides) : side;
          if (!MATERIALS || ts >= 0) offer_first(m, t, k, r, dlen, ts, near_d, far_d, best);
        }
        if (__ballot_sync(full, leaf)) {
          lim_hit = slab_limit(warp_min((best.t + best.err) * (1.0f + kSlabMargin)));
          lim = fminf(lim, lim_hit);
        }
        if (__ballot_sync(full, enter)) wide_push(stack, sp, lane, enter, link, key, key);
      }
    }
    for (int x = 1; x < 32; x <<= 1) {
      Best o;
      o.t = __shfl_xor_sync(full, best.t, x);
      o.err = __shfl_xor_sync(full, best.err, x);
      o.rec = __shfl_xor_sync(full, best.rec, x);
      if (o.rec != 0xFFFFFFFFu && o.rec != best.rec && !(o.t - o.err > best.t + best.err)) {
        if (o.t + o.err < best.t - best.err) best = o;
        else  // both are hits: the side, near and far of the call hold for them
          best = offer_slow(m.tris, o.rec, r.o, r.d, kSideDouble, 0.0f, kInf, best);
      }
    }
    // the record, complete: with few rays the finalize kernel's launch would cost more than it saves
    if (lane == 0) finish_first(m, best.rec, r, out + rid);
  }
}

__global__ void __launch_bounds__(kBlock) closest_point_wide_kernel(MeshDev m, const float* __restrict__ pts, uint32_t n,
                                                                    float max_t, bvhc_closest* __restrict__ out,
                                                                    int cap) {
  extern __shared__ uint2 s_stack[];
  __shared__ uint2 s_tie[kClosestTies][kBlock];
  const unsigned lane = threadIdx.x & 31u;
  uint2* stack = s_stack + (threadIdx.x >> 5) * cap;
  const MaxThreshold mx = max_threshold(max_t);
  for (uint32_t qid = blockIdx.x * kWarps + (threadIdx.x >> 5); qid < n; qid += gridDim.x * kWarps) {
    const float* q = pts + 3 * (size_t)qid;
    const float3 p = make_float3(__ldg(q), __ldg(q + 1), __ldg(q + 2));
    // a point that is not finite reaches no leaf
    const bool finite = fabsf(p.x) <= FLT_MAX && fabsf(p.y) <= FLT_MAX && fabsf(p.z) <= FLT_MAX;
    Nearest best = nearest_none();
    if (finite && m.n_roots > 0) {
      if (lane == 0) stack[0] = make_uint2(m.quad_roots[0], 0u);
      __syncwarp();
      closest_walk_wide(m, p, mx, stack, kWideSpare, 1, 0, FLT_MAX, best, s_tie);
    }
    store_merged<32>(m.tris, p, best, true, reinterpret_cast<uint32_t*>(out + qid), s_tie);
  }
}

}  // namespace dev

cudaError_t launch_raycast_first_wide(const MeshDev& m, const BatchDev* batch, const float* rays, uint64_t n, int side,
                                      const SideTable& sides, float near_d, float far_d, bvhc_hit* out,
                                      cudaStream_t stream, const uint32_t* queue, const unsigned int* qcount) {
  const int cap = dev::wide_stack(group_stack(m));
  const size_t smem = wide_smem(group_stack(m));
  auto kernel = sides.per_material ? dev::raycast_first_wide_kernel<true> : dev::raycast_first_wide_kernel<false>;
  const BatchDev bd = batch ? *batch : BatchDev{nullptr, nullptr, 0};
  const unsigned int grid = (unsigned int)((n + dev::kWarps - 1) / dev::kWarps);
  kernel<<<grid, dev::kBlock, smem, stream>>>(m, bd, batch != nullptr, rays, (uint32_t)n, side, sides, near_d, far_d,
                                              dev::ranged(near_d, far_d), out, queue, qcount, cap);
  return cudaGetLastError();
}

cudaError_t launch_closest_wide(const MeshDev& m, const float* pts, uint32_t n, float max_t, bvhc_closest* out,
                                cudaStream_t stream) {
  const int cap = dev::wide_stack(group_stack(m));
  const size_t smem = wide_smem(group_stack(m));
  const unsigned int grid = std::min((n + dev::kWarps - 1) / dev::kWarps, (unsigned int)sm_count() * 8u);
  dev::closest_point_wide_kernel<<<grid, dev::kBlock, smem, stream>>>(m, pts, n, max_t, out, cap);
  return cudaGetLastError();
}

}  // namespace bvhc
