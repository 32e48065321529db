// Device-resident layout of a MeshBVH, shared by the host re-layout code and the kernels.
//
// The serialized reference node (src/core/build/buildUtils.js:31-92) is 32 bytes: its own box
// plus either (right-child offset, split axis) or (triangle offset, count, leaf flag).  A query
// visiting an internal node always reads BOTH children's boxes (intersectsNodeBounds on c1 and
// c2, or both shapecast scores), so the device layout stores, per internal node, one 64-byte
// "child pair" record holding the two child boxes and the two child links.  One visit is then
// one 64-byte, 64-byte-aligned read (two 32-byte sectors), instead of two scattered 32-byte
// reads.  The root's own box is never tested by the reference and is not stored.
//
// Leaf triangles are copied into 48-byte records in DFS leaf order, vertices inline, so that a
// leaf is one contiguous run of 16-byte-aligned loads and needs no index indirection.
#pragma once

#include <math.h>

#include <cstdint>

namespace bvhc {

// Child link: internal child -> child-pair record index; leaf child -> kLeafBit | first
// triangle record; an empty leaf -> kEmptyLeaf.
constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kEmptyLeaf = 0xFFFFFFFFu;
constexpr int kMaxStack = 64;  // deepest supported tree (the reference's default maxDepth is 40)

struct alignas(64) PairNode {
  // f[0..5]  left child  box (min xyz, max xyz)
  // f[6..11] right child box
  float f[12];
  uint32_t link[2];   // left, right child links
  uint32_t axis;      // split axis of this node (0, 1, 2)
  uint32_t flags;     // 0 (reserved)
};
static_assert(sizeof(PairNode) == 64, "PairNode must be 64 bytes");

// Four-child record of the ray queries, collapsed from the child-pair tree (each internal child
// replaced in place by its own two children, largest surface area first, until there are four
// children or only leaves; the children stay in the tree's left-to-right order).  A child is one
// 32-byte sector (one 256-bit load): its box as centre and half extent, x and y side by side as the
// operands of packed float instructions.  With centre and half extent a slab's entry and exit are
// t_c -+ r, additions on the FMA pipe, where lo / hi planes need a minimum and a maximum per axis on
// the half-rate ALU pipe.  The half extents are rounded up (box_centre_half), so the box holds the
// reference's.  Unused children have link kEmptyLeaf and a NaN box, which no ray enters.  Every root is
// a record: a root that is a leaf is one child with an unbounded box.
struct alignas(32) QuadChild {
  float c[2], h[2];   // x, y
  float cz, hz;
  uint32_t link;      // internal child -> quad record index; else a run of triangle records (run_link)
  uint32_t count;     // a part of a leaf (or a root that is one): its triangle records, else 0
};
struct alignas(128) QuadNode {
  QuadChild c[4];
};
static_assert(sizeof(QuadNode) == 128, "QuadNode must be 128 bytes");

// What a child of a four-child record is made from: its link and count, and where its box comes from: the
// child-pair slot (2 * pair + side), or kLeafBit | the first of its `count` triangle records; kEmptyLeaf: unused,
// or with another link a root leaf's unbounded box.
struct QuadShape {
  uint32_t link, count, src;
};

// A child pair in the same form, for the warp-shared ray traversals: the two children of a PairNode and,
// in c[0].count, its split axis (an empty leaf's box is NaN).
struct alignas(64) RayPair {
  QuadChild c[2];
};
static_assert(sizeof(RayPair) == 64, "RayPair must be 64 bytes");

// The four-child record for closestPointToPoint, whose maxThreshold is decided on the reference's exact
// boxes: lo / hi bounds, an unused child at infinity.
struct alignas(32) BoxChild {
  float lo[3], hi[3];
  uint32_t link, part;  // as QuadChild's link and count
};
struct alignas(128) BoxNode {
  BoxChild c[4];
};
static_assert(sizeof(BoxNode) == 128, "BoxNode must be 128 bytes");

constexpr float kBoxUnbounded = 3e38f;

// A leaf of a four-child record: a run of at most kMaxRun consecutive triangle records of one of the
// tree's leaves (a larger leaf has a record, or several, of parts with their own exact bounds), as
// kLeafBit, the run's length less one in two bits, its first record in the rest.
constexpr int kMaxRun = 4;
constexpr int kRunShift = 29;
constexpr uint32_t kRunFirst = (1u << kRunShift) - 1u;
#ifdef __CUDACC__
__host__ __device__
#endif
    inline uint32_t run_link(uint32_t first, int count) {
  return kLeafBit | ((uint32_t)(count - 1) << kRunShift) | first;
}

#ifdef __CUDACC__
__host__ __device__
#endif
    // One axis of a box as centre and half extent.  The half extent reaches the farther bound (a difference
    // of float32 values, rounded once) and carries 64u of itself, u = 2^-24, for the ray test (traverse.cuh's
    // slab_axis), or more where that is lost below 2^-126.  Swapped bounds count as the box between them, as
    // in the slab test with minimum and maximum; bounds that are not numbers, or too large, give an
    // unbounded axis.
    inline void box_centre_half(float lo, float hi, float& c, float& h) {
  c = 0.5f * lo + 0.5f * hi;
  const float a = hi - c, b = c - lo;
  const float aa = a < 0.0f ? -a : a, ab = b < 0.0f ? -b : b;
  h = (aa > ab ? aa : ab) * (1.0f + 3.814697265625e-06f) + 7.174648137343064e-43f;
  if (!(aa < kBoxUnbounded && ab < kBoxUnbounded && h < kBoxUnbounded)) {
    c = 0.0f;
    h = kBoxUnbounded;
  }
}

struct alignas(16) TriRecord {
  // v[0..8] = a.xyz, b.xyz, c.xyz ; face = reference faceIndex ; flags bit 0 = last in leaf ;
  // material = materialIndex of the geometry group holding the triangle (kNoMaterial: none)
  float v[9];
  uint32_t face;
  uint32_t flags;
  uint32_t material;
};
static_assert(sizeof(TriRecord) == 48, "TriRecord must be 48 bytes");

constexpr uint32_t kTriLast = 1u;
constexpr uint32_t kNoMaterial = 0xFFFFFFFFu;
constexpr int kMaxMaterials = 64;

#ifdef __CUDACC__
__host__ __device__
#endif
    // A child of a four-child record; b (lo, hi) gets its box, which is that of its child-pair slot, or for a
    // part of a leaf the bounds of its triangles.
    inline QuadChild quad_child(const QuadShape& s, const PairNode* pairs, const TriRecord* tris, float* b) {
  QuadChild c;
  c.link = s.link;
  c.count = s.count;
  if (s.src == kEmptyLeaf) {
    const bool unused = s.link == kEmptyLeaf;
    for (int a = 0; a < 3; ++a) {
      b[a] = unused ? INFINITY : -INFINITY;
      b[3 + a] = INFINITY;
    }
    c.c[0] = c.c[1] = c.cz = unused ? NAN : 0.0f;
    c.h[0] = c.h[1] = c.hz = unused ? NAN : kBoxUnbounded;
    return c;
  }
  if (!(s.src & kLeafBit)) {
    const float* f = pairs[s.src >> 1].f + 6 * (s.src & 1u);
    for (int a = 0; a < 6; ++a) b[a] = f[a];
  } else {
    const TriRecord* t = tris + (s.src & ~kLeafBit);
    for (int a = 0; a < 3; ++a) b[a] = b[3 + a] = t->v[a];
    for (uint32_t q = 0; q < s.count; ++q)
      for (int a = 0; a < 9; ++a) {
        b[a % 3] = fminf(b[a % 3], t[q].v[a]);
        b[3 + a % 3] = fmaxf(b[3 + a % 3], t[q].v[a]);
      }
  }
  box_centre_half(b[0], b[3], c.c[0], c.h[0]);
  box_centre_half(b[1], b[4], c.c[1], c.h[1]);
  box_centre_half(b[2], b[5], c.cz, c.hz);
  return c;
}

// Per-call side selection: a single side for every triangle, or one side per material.
struct SideTable {
  int8_t side[kMaxMaterials];
  int32_t n;        // number of materials
  int32_t per_material;
};

}  // namespace bvhc
