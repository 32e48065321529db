// A stand-in for the CUDA runtime and for the launches that the handle code (csrc/api.cu) makes, over host
// memory, for CPU tests of that code: allocations that fail on request, a count of what is held, and checks of
// what each launch is given (test infrastructure; compiled by tests/test_handles_cpu.py).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>

#include "kernels.cuh"

namespace {
std::map<void*, size_t> held;
int fail_in = 0;  // > 0: that many allocations from now, one fails
int bad = 0;      // launches given records that do not belong together
int packets = 0;
int host_blocks = 0;  // page-locked allocations so far
bool host_gone = false;  // their context is

bool live(const void* p, size_t bytes) {
  auto it = held.find(const_cast<void*>(p));
  return it != held.end() && it->second >= bytes;
}
void check(bool ok) { bad += !ok; }
}  // namespace

extern "C" {
void fake_fail_in(int n) { fail_in = n; }
int fake_fail_left() { return fail_in; }
int64_t fake_held() { return (int64_t)held.size(); }
int fake_bad() { return bad; }
int fake_packets() { return packets; }
int fake_host_blocks() { return host_blocks; }
void fake_lose_host(int gone) { host_gone = gone != 0; }

cudaError_t cudaMalloc(void** p, size_t n) {
  if (fail_in > 0 && --fail_in == 0) return cudaErrorMemoryAllocation;
  *p = std::malloc(n ? n : 1);
  held[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  auto it = held.find(p);
  check(it != held.end());
  if (it == held.end()) return cudaErrorInvalidValue;
  std::memset(p, 0xDD, it->second);
  held.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  ++host_blocks;
  return cudaMalloc(p, n);
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = host_gone ? cudaMemoryTypeUnregistered : cudaMemoryTypeHost;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
}

namespace bvhc {

cudaError_t launch_ray_pairs(const PairNode* pairs, uint64_t n, RayPair* out, cudaStream_t) {
  check(live(pairs, n * sizeof(PairNode)) && live(out, n * sizeof(RayPair)));
  for (uint64_t k = 0; k < n; ++k)
    for (int s = 0; s < 2; ++s) out[k].c[s].link = pairs[k].link[s];
  return cudaSuccess;
}

cudaError_t launch_quad_boxes(QuadNode* quads, uint64_t n, const QuadShape* shape, const PairNode* pairs,
                              const TriRecord* tris, BoxNode*, cudaStream_t) {
  check(live(quads, n * sizeof(QuadNode)) && live(shape, 4 * n * sizeof(QuadShape)));
  auto p = held.find(const_cast<PairNode*>(pairs)), t = held.find(const_cast<TriRecord*>(tris));
  check(p != held.end() && t != held.end());
  if (p == held.end() || t == held.end()) return cudaErrorInvalidValue;
  float box[6];
  for (uint64_t k = 0; k < 4 * n; ++k) {
    const QuadShape& s = shape[k];
    const bool in = s.src == kEmptyLeaf || (s.src & kLeafBit ? (s.src & ~kLeafBit) + s.count <= t->second / sizeof(TriRecord)
                                                             : s.src / 2 < p->second / sizeof(PairNode));
    check(in);
    if (in) quads[k / 4].c[k % 4] = quad_child(s, pairs, tris, box);
  }
  return cudaSuccess;
}

cudaError_t launch_refit(const RefitPlan& plan, PairNode* pairs, RayPair* rays, TriRecord* tris, const uint32_t*,
                         const float*, int, bool, cudaStream_t) {
  check(live(rays, plan.n_pairs * sizeof(RayPair)) && live(plan.arrive, 8 * plan.n_pairs));
  check(live(pairs, plan.n_pairs * sizeof(PairNode)) && live(plan.leaves, plan.n_leaves * sizeof(RefitLeaf)));
  for (uint32_t k = 0; k < plan.n_leaves; ++k) {  // each leaf's run ends where the records say
    const RefitLeaf& l = plan.leaves[k];
    if (l.count) check((tris[l.first + l.count - 1].flags & kTriLast) && (l.slot & kRootSlot || l.slot / 2 < plan.n_pairs));
  }
  return cudaSuccess;
}

cudaError_t launch_raycast_first_packet(const MeshDev& m, const float*, uint64_t, int, const SideTable&, float, float,
                                        bvhc_hit*, const TraversalConfig&, cudaStream_t, uint32_t*, unsigned int*,
                                        const RaySort*) {
  ++packets;
  auto it = held.find(const_cast<PairNode*>(m.nodes));
  const bool ok = it != held.end() && m.ray_pairs && live(m.ray_pairs, it->second / sizeof(PairNode) * sizeof(RayPair));
  check(ok);
  if (ok)
    for (size_t k = 0; k < it->second / sizeof(PairNode); ++k)
      for (int s = 0; s < 2; ++s) check(m.ray_pairs[k].c[s].link == m.nodes[k].link[s]);
  auto q = held.find(const_cast<QuadNode*>(m.quads)), t = held.find(const_cast<TriRecord*>(m.tris));
  check(q != held.end() && t != held.end());
  if (q != held.end() && t != held.end())
    for (size_t k = 0; k < q->second / sizeof(QuadNode); ++k)
      for (const QuadChild& c : m.quads[k].c) {
        if (c.link == kEmptyLeaf) continue;
        if (c.link & kLeafBit) check((c.link & kRunFirst) + (c.link >> kRunShift & 3u) < t->second / sizeof(TriRecord));
        else check(c.link < q->second / sizeof(QuadNode));
      }
  return cudaSuccess;
}

}  // namespace bvhc
