// raycastFirst, warp-cooperative forms (over child pairs, in queue, input or tiled ray order, and
// over four-child records); and their launch.
#include <algorithm>

#include "traverse.cuh"

namespace bvhc {
namespace dev {

// ---------------------------------------------------------------------------------------------
// raycastFirst, warp-cooperative form for coherent rays (camera rays in pixel order).  The 32
// rays of a warp walk the tree together with one shared stack: every child pair is fetched once
// for the warp (a broadcast load), each lane tests it against its own ray, and the warp enters a
// child if any lane's ray enters it (nearest first by majority vote).  A leaf is tested by all
// lanes at once, so the triangle tests run at full SIMD width.  Each lane keeps its own entry
// distance for every stacked child; a stacked child is skipped when no lane still needs it.
// Visiting a node a lane's ray does not enter costs that lane nothing but idle time, and testing
// a triangle it would not have reached cannot change its closest hit.  The kernel leaves each hit
// pending (its triangle record); finalize_first_kernel computes the reported records, which keeps
// the float-float record code out of the traversal kernel.
// The kernel is bound by issued instructions.  A node's two boxes are read as centre and half extent
// (RayPair: 13 instructions a box, 5 of them on the half-rate ALU pipe, against 31 and 19 with lo / hi
// planes), the ray's limit changes at leaves only, and with ORDER 0 the warp's majority per axis is
// taken once: 2^24 camera rays on the 2M-triangle knot 3724 -> 3204 us.
// ---------------------------------------------------------------------------------------------

// BLOCK threads per block (64, 128 or 256), STACK shared-stack entries (32 or 64; the launch picks 32
// only for trees shallow enough that no traversal can need more).
template <int ORDER, int MINB, int BLOCK, int STACK>
__global__ void __launch_bounds__(BLOCK, MINB) raycast_first_packet_kernel(MeshDev m, const float* __restrict__ rays,
                                                                     uint64_t n, int side, const SideTable sides,
                                                                     float near_d, float far_d,
                                                                     bvhc_hit* __restrict__ out,
                                                                     const uint32_t* __restrict__ queue,
                                                                     const unsigned int* __restrict__ qcount,
                                                                     uint64_t pitch, int rows_log2) {
  __shared__ uint32_t s_link[BLOCK / 32][STACK];
  const unsigned full = 0xFFFFFFFFu;
  const int w = threadIdx.x >> 5;
  const unsigned lane = threadIdx.x & 31u;
  // with a queue (root-box pre-pass, optionally sorted) a warp takes 32 consecutive queue entries;
  // without one, 32 consecutive rays or (pitch > 0) a tile of them
  const uint64_t n_work = queue ? (uint64_t)__ldg(qcount) : n;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if ((uint64_t)blockIdx.x * blockDim.x >= n_work) return;  // block-uniform
  const bool valid = i < n_work;
  if (valid && queue) i = __ldg(queue + i);
  else if (valid && pitch) i = tiled_index(i, pitch, rows_log2, n);
  RayF r;
  float dlen = 1.0f;
  if (valid) {
    r = make_ray(rays, i);
    dlen = sqrtf(r.d.x * r.d.x + r.d.y * r.d.y + r.d.z * r.d.z);
  } else {
    r.o = make_float3(0.f, 0.f, 0.f);
    r.d = make_float3(1.f, 0.f, 0.f);
    r.inv = make_float3(1.f, 1e30f, 1e30f);
    r.dk = kFilterK;
  }
  const RaySlab rs = ray_slab(r);
  const float near_s = slab_near(near_d);
  // a lane without a ray enters nothing
  const float far_s = valid ? slab_far(far_d) : -kInf;
  float lim_hit = valid ? kInf : -kInf, lim = far_s;
  // ORDER 0: per axis, whether most of the warp's rays go towards larger coordinates
  const int half = (__popc(__ballot_sync(full, valid)) + 1) / 2;
  const unsigned forward = (__popc(__ballot_sync(full, valid && r.d.x >= 0.0f)) >= half ? 1u : 0u) |
                           (__popc(__ballot_sync(full, valid && r.d.y >= 0.0f)) >= half ? 2u : 0u) |
                           (__popc(__ballot_sync(full, valid && r.d.z >= 0.0f)) >= half ? 4u : 0u);
  Best best{kInf, 0.0f, 0xFFFFFFFFu};
  const float kNo = __int_as_float(0x7FFFFFFF);  // NaN: this lane does not want the entry
  float lane_t[STACK];
  for (int root = 0; root < m.n_roots; ++root) {
    uint32_t link = m.roots[root];
    int sp = 0;
    for (;;) {
      bool pop = false;
      if (link & kLeafBit) {
        if (link != kEmptyLeaf && valid) {
          leaf_first(m, link & ~kLeafBit, r, dlen, side, sides, near_d, far_d, best);
          lim_hit = slab_limit((best.t + best.err) * (1.0f + kSlabMargin));
          lim = fminf(far_s, lim_hit);
        }
        pop = true;
      } else {
        const RayPair* rp = m.ray_pairs + link;
        const ChildBox c0 = load_child(rp->c), c1 = load_child(rp->c + 1);
        float e0, e1;
        const bool h0 = child_hit(c0, rs, near_s, lim, e0), h1 = child_hit(c1, rs, near_s, lim, e1);
        const unsigned b0 = __ballot_sync(full, h0), b1 = __ballot_sync(full, h1);
        if (b0 && b1) {
          const bool left_wins = ORDER == 0 ? (forward >> c0.part) & 1u
                                            : __popc(__ballot_sync(full, valid && e0 <= e1)) >= half;
          if (sp >= STACK) {
            if (lane == 0) atomicOr(m.err, kErrStackOverflow);
            best.rec = 0xFFFFFFFFu;
            root = m.n_roots;
            break;
          }
          if (lane == 0) s_link[w][sp] = left_wins ? c1.link : c0.link;
          lane_t[sp] = left_wins ? (h1 ? e1 : kNo) : (h0 ? e0 : kNo);
          ++sp;
          link = left_wins ? c0.link : c1.link;
          __syncwarp();
        } else if (b0) {
          link = c0.link;
        } else if (b1) {
          link = c1.link;
        } else {
          pop = true;
        }
      }
      if (pop) {
        bool found = false;
        while (sp > 0) {
          --sp;
          if (__ballot_sync(full, lane_t[sp] <= lim_hit)) {
            link = s_link[w][sp];
            found = true;
            break;
          }
        }
        if (!found) break;
      }
    }
  }
  if (valid) store_first_pending(out + i, best);  // finalize_first_kernel completes a hit
}

// ---------------------------------------------------------------------------------------------
// raycastFirst, warp-cooperative over the four-child records (m.quads): the same shared traversal
// as above with half as many node visits.  At a record each lane tests the four child boxes; the
// children any lane enters are ordered by the entry distances of the first lane that enters one (the warp's rays are coherent), the nearest is
// visited and the others are stacked farthest first, each with every lane's own entry distance.
// ---------------------------------------------------------------------------------------------
template <int MINB>
__global__ void __launch_bounds__(kBlock, MINB) raycast_first_packet4_kernel(
    MeshDev m, const float* __restrict__ rays, uint64_t n, int side, const SideTable sides, float near_d,
    float far_d, bvhc_hit* __restrict__ out, const uint32_t* __restrict__ queue,
    const unsigned int* __restrict__ qcount, uint64_t pitch, int rows_log2, bool ranged_call) {
  __shared__ uint32_t s_link[kWarps][kMaxStack];
  const unsigned full = 0xFFFFFFFFu;
  const int w = threadIdx.x >> 5;
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t n_work = queue ? (uint64_t)__ldg(qcount) : n;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if ((uint64_t)blockIdx.x * blockDim.x >= n_work) return;  // block-uniform
  const bool valid = i < n_work;
  if (valid && queue) i = __ldg(queue + i);
  else if (valid && pitch) i = tiled_index(i, pitch, rows_log2, n);
  RayF r;
  float dlen = 1.0f;
  if (valid) {
    r = make_ray(rays, i);
    dlen = sqrtf(r.d.x * r.d.x + r.d.y * r.d.y + r.d.z * r.d.z);
  } else {
    r.o = make_float3(0.f, 0.f, 0.f);
    r.d = make_float3(1.f, 0.f, 0.f);
    r.inv = make_float3(1.f, 1e30f, 1e30f);
    r.dk = kFilterK;
  }
  const RaySlab rs = ray_slab(r);
  const float near_s = slab_near(near_d);
  const bool odd = ranged_call && free_parts(r.d, near_d);  // parts of leaves are not held against near and far
  Best best{kInf, 0.0f, 0xFFFFFFFFu};
  float lane_t[kMaxStack];
  for (int root = 0; root < m.n_roots; ++root) {
    uint32_t link = m.quad_roots[root];
    int sp = 0;
    for (;;) {
      bool pop = false;
      if (link & kLeafBit) {
        if (valid) run_first(m, link, r, dlen, side, sides, near_d, far_d, best);
        pop = true;
      } else {
        // the record's four children: one 256-bit load each
        ChildBox ch[4];
        uint32_t ck[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          ch[c] = load_child(m.quads[link].c + c);
          ck[c] = ch[c].link;
        }
        const float lim_hit = slab_limit((best.t + best.err) * (1.0f + kSlabMargin));
        const float lim = fminf(slab_far(far_d), lim_hit);
        float e[4];
        bool h[4];
        unsigned b[4];
        unsigned any = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const bool free_box = odd && ch[c].part;
          h[c] = child_hit(ch[c], rs, free_box ? 0.0f : near_s, free_box ? lim_hit : lim, e[c]) && valid;
          b[c] = __ballot_sync(full, h[c]);
          any |= b[c];
        }
        if (!any) {
          pop = true;
        } else {
          const int leader = __ffs(any) - 1;
          float key[4];
          int idx[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float kc = __shfl_sync(full, h[c] ? e[c] : kInf, leader);
            key[c] = b[c] ? kc : kInf;
            idx[c] = c;
          }
          // sort the four (key, child) pairs, nearest first (warp-uniform values)
          auto cas = [&](int a, int c) {
            if (key[c] < key[a]) {
              float tk = key[a]; key[a] = key[c]; key[c] = tk;
              int ti = idx[a]; idx[a] = idx[c]; idx[c] = ti;
            }
          };
          cas(0, 1); cas(2, 3); cas(0, 2); cas(1, 3); cas(1, 2);
          if (sp + 3 > kMaxStack) {
            if (lane == 0) atomicOr(m.err, kErrStackOverflow);
            best.rec = 0xFFFFFFFFu;
            root = m.n_roots;
            break;
          }
          // children that some lane enters, farthest pushed first; the nearest is visited now
          uint32_t next = kEmptyLeaf;
          bool have_next = false;
#pragma unroll
          for (int j = 3; j >= 0; --j) {
            const int c = idx[j];
            if (!b[c]) continue;
            if (j == 0) {
              next = ck[c];
              have_next = true;
            } else {
              if (lane == 0) s_link[w][sp] = ck[c];
              lane_t[sp] = h[c] ? e[c] : kInf;
              ++sp;
            }
          }
          if (have_next) {
            link = next;
          } else {  // the first key belonged to a child no lane enters: every entered one was stacked
            pop = true;
          }
          __syncwarp();
        }
      }
      if (pop) {
        bool found = false;
        while (sp > 0) {
          --sp;
          float plim = slab_limit((best.t + best.err) * (1.0f + kSlabMargin));
          if (__ballot_sync(full, valid && lane_t[sp] <= plim)) {
            link = s_link[w][sp];
            found = true;
            break;
          }
        }
        if (!found) break;
      }
    }
  }
  if (valid) store_first_pending(out + i, best);  // finalize_first_kernel completes a hit
}

}  // namespace dev

template <int BLOCK, int STACK>
static void launch_packet_kernel(const MeshDev& m, const float* rays, uint64_t n, int side, const SideTable& sides,
                                 float near_d, float far_d, bvhc_hit* out, int order, int occupancy,
                                 cudaStream_t stream, const uint32_t* queue, const unsigned int* qcount,
                                 uint64_t pitch, int rows_log2) {
  // occupancy 1 / 2 ask for 768 / 1024 resident threads per SM whatever the block size
  constexpr int k6 = 6 * 128 / BLOCK, k8 = 8 * 128 / BLOCK;
  auto kernel = order == 0 ? (occupancy == 0   ? dev::raycast_first_packet_kernel<0, 1, BLOCK, STACK>
                              : occupancy == 1 ? dev::raycast_first_packet_kernel<0, k6, BLOCK, STACK>
                                               : dev::raycast_first_packet_kernel<0, k8, BLOCK, STACK>)
                           : (occupancy == 0   ? dev::raycast_first_packet_kernel<1, 1, BLOCK, STACK>
                              : occupancy == 1 ? dev::raycast_first_packet_kernel<1, k6, BLOCK, STACK>
                                               : dev::raycast_first_packet_kernel<1, k8, BLOCK, STACK>);
  const unsigned int grid = (unsigned int)((n + BLOCK - 1) / BLOCK);
  kernel<<<grid, BLOCK, 0, stream>>>(m, rays, n, side, sides, near_d, far_d, out, queue, qcount, pitch, rows_log2);
}

cudaError_t launch_raycast_first_packet(const MeshDev& m, const float* rays, uint64_t n, int side,
                                        const SideTable& sides, float near_d, float far_d, bvhc_hit* out,
                                        const TraversalConfig& cfg, cudaStream_t stream, uint32_t* queue,
                                        unsigned int* qcount, const RaySort* sort) {
  if (n == 0) return cudaSuccess;
  if (!m.ray_pairs) return cudaErrorInvalidValue;
  const bool compact = queue != nullptr && qcount != nullptr && n < (1ull << 32);
  if (compact) {
    cudaError_t e = prepare_queue(m, nullptr, rays, n, near_d, far_d, out, queue, qcount, sort, stream);
    if (e != cudaSuccess) return e;
  } else {
    queue = nullptr;
    qcount = nullptr;
  }
  // the tiled order applies to the whole ray range (a queue is already in its own order)
  const int rl = tile_rows_log2(cfg.tile_rows);
  const uint64_t pitch = (!queue && cfg.tile >= 8 && cfg.tile % (32 >> rl) == 0) ? (uint64_t)cfg.tile : 0;
  // the four-child form stacks up to three children a step, and gives up where three no longer fit
  if (cfg.wide && m.quads && m.quad_roots && m.quad_stack + 3 <= kMaxStack) {
    auto k4 = cfg.occupancy == 0   ? dev::raycast_first_packet4_kernel<1>
              : cfg.occupancy == 1 ? dev::raycast_first_packet4_kernel<6>
                                   : dev::raycast_first_packet4_kernel<8>;
    k4<<<grid_for(n), dev::kBlock, 0, stream>>>(m, rays, n, side, sides, near_d, far_d, out, queue, qcount, pitch,
                                                rl, dev::ranged(near_d, far_d));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_finalize_first(m, rays, n, out, queue, qcount, stream);
  }
  const bool s32 = stack_entries(m, cfg.stack) == 32;
  const int block = cfg.block == 64 || cfg.block == 256 ? cfg.block : 128;
#define BVHC_PACKET(B, S) \
  launch_packet_kernel<B, S>(m, rays, n, side, sides, near_d, far_d, out, cfg.order, cfg.occupancy, stream, queue, \
                             qcount, pitch, rl)
  if (block == 64) {
    if (s32) BVHC_PACKET(64, 32);
    else BVHC_PACKET(64, 64);
  } else if (block == 256) {
    if (s32) BVHC_PACKET(256, 32);
    else BVHC_PACKET(256, 64);
  } else {
    if (s32) BVHC_PACKET(128, 32);
    else BVHC_PACKET(128, 64);
  }
#undef BVHC_PACKET
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_finalize_first(m, rays, n, out, queue, qcount, stream);
}

}  // namespace bvhc
