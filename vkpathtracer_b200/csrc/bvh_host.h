// bvh_host.h -- host side of the acceleration structure: primitive flattening,
// the binary midpoint BVH, and its collapse into the 128-byte wide-node layout
// that the sm_100a traversal kernels read from HBM.
#pragma once

#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include "bvh_layout.h"

namespace vkptc {

struct HostPrim {
  float v0[3], e1[3], e2[3], n[3];
  uint32_t material;
};

struct BinNode {
  float lo[3], hi[3];
  int32_t left, right, first, count;
};

// Wide node: six float4 of child bounds (lo.x[4], hi.x[4], lo.y[4], hi.y[4],
// lo.z[4], hi.z[4]: the node test takes its near and far planes by the ray's
// signs), then int4 child refs, then int4 meta (x = valid child count).  Child ref >= 0: wide node index; < 0: leaf,
// ~ref = (first_triangle << 3) | (count - 1); kEmptyChild: an unused slot
// (so the traversal needs no child count).  128 bytes, one cache line.
struct alignas(16) WideNode {
  float lox[4], hix[4], loy[4], hiy[4], loz[4], hiz[4];
  int32_t child[4];
  int32_t meta[4];
};
static_assert(sizeof(WideNode) == 128, "wide node must be one 128-byte line");

#ifdef __CUDACC__
#define VKPTC_HD __host__ __device__
#else
#define VKPTC_HD
#endif

// Child k's box: the binary node's bounds.  From 1024 on, where the padding of
// 1e-4 is an ulp or nothing, the upper ones are an ulp or two higher: a ray with
// a component of 0 along an upper face (the surface itself there) would get the
// far distance 0 from the node test, and the reference counts it as inside.
VKPTC_HD inline float UpperFace(float hi) {
  const float a = hi < 0.0f ? -hi : hi;
  return a >= 1024.0f ? hi + a * 1.1920928955078125e-7f : hi;   // 2^-23
}
VKPTC_HD inline void SetWideSlot(WideNode& n, int k, const float* lo, const float* hi) {
  n.lox[k] = lo[0];
  n.loy[k] = lo[1];
  n.loz[k] = lo[2];
  n.hix[k] = UpperFace(hi[0]);
  n.hiy[k] = UpperFace(hi[1]);
  n.hiz[k] = UpperFace(hi[2]);
}
// The wide collapse.  A wide node takes up to four subtrees of the binary tree
// as its slots, chosen bottom-up for the least expected cost (area times work):
// cost(i) of a subtree is that of at most i roots for it, where one root is a
// leaf of all its triangles (at most 8; see CollapseNode) or a wide node over its
// best four (the dynamic programme of Ylitie, Karras and Laine, "Efficient
// Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs", HPG 2017, 3.1).
// Opening the largest slot greedily, top-down, filled 3.05 of 4 slots on the
// 1,046,904-triangle sphere and kept the binary tree's leaves.
// Choosing it this way makes 31 % fewer wide nodes there; rays from hit points
// 2.57 -> 2.66 G/s, random rays 4.18 -> 4.63, camera rays 4.31 -> 4.22; in the
// closed box 11.5 -> 12.2 G/s; the 64-job batch 523.6 -> 510.5 ms.  Triangle costs of
// 0.3 and 0.9 (and binary leaves of one triangle) were within 3 % either way.
constexpr float kTriangleCost = 0.6f;   // a triangle test against a node's four box tests
constexpr int32_t kWideLeafMax = 8;     // triangles in a leaf (the ref has three bits for it)
// A subtree's choices in one byte: bit 0: one root is a leaf; bits 1-3: two, three,
// four roots are no better than one fewer; bits 4-5, 6-7: the left child's roots
// when three, four are split (of two, one each).
VKPTC_HD inline bool CollapseLeaf(uint32_t bits) { return (bits & 1u) != 0u; }
// Roots of the left child when the subtree takes i = 2..4 of its own.
VKPTC_HD inline uint32_t CollapseSplit(uint32_t bits, uint32_t i) {
  return i == 2u ? 1u : (i == 3u ? (bits >> 4) & 3u : (bits >> 6) & 3u);
}
VKPTC_HD inline bool CollapseFewer(uint32_t bits, uint32_t i) { return ((bits >> (i - 1u)) & 1u) != 0u; }
VKPTC_HD inline float HalfArea(const float* lo, const float* hi) {
  const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
  return dx * dy + dy * dz + dz * dx;
}
// Costs and choices of an internal node from its children's; plain float
// arithmetic, so the host and the device collapse choose the same.  merge: the
// subtree may become one leaf.  Not in the reference's own tree: a triangle whose
// distance is badly conditioned can be hit outside its box, so one that the
// reference's leaf box culls must not be tested under the box of several leaves.
VKPTC_HD inline uint32_t CollapseNode(const float* l, const float* r, float area, int32_t count, bool merge,
                                     float* out) {
  const float d2 = l[0] + r[0];
  const float a3 = l[0] + r[1], b3 = l[1] + r[0];
  const float d3 = b3 < a3 ? b3 : a3;
  const float a4 = l[0] + r[2], b4 = l[1] + r[1], c4 = l[2] + r[0];
  uint32_t k4 = 1u;
  float d4 = a4;
  if (b4 < d4) {
    d4 = b4;
    k4 = 2u;
  }
  if (c4 < d4) {
    d4 = c4;
    k4 = 3u;
  }
  uint32_t bits = ((b3 < a3 ? 2u : 1u) << 4) | (k4 << 6);
  const float node = area + d4, leaf = area * (kTriangleCost * static_cast<float>(count));
  const bool is_leaf = merge && count <= kWideLeafMax && !(node < leaf);
  out[0] = is_leaf ? leaf : node;
  if (is_leaf) bits |= 1u;
  const float d[3] = {d2, d3, d4};
  for (int i = 0; i < 3; ++i) {
    const bool fewer = !(d[i] < out[i]);
    out[i + 1] = fewer ? out[i] : d[i];
    if (fewer) bits |= 2u << i;
  }
  return bits;
}

// An unused slot: no box (its ref, kEmptyChild, is what the traversal tests).
VKPTC_HD inline void ClearWideSlot(WideNode& n, int k) {
  n.lox[k] = n.loy[k] = n.loz[k] = 1.0f;
  n.hix[k] = n.hiy[k] = n.hiz[k] = -1.0f;
  n.child[k] = kEmptyChild;
}

// Triangle record in leaf order: v0, e1, e2, then the reference primitive
// index, the binary leaf that holds it and its lane in that leaf (the last
// two resolve exact-distance ties in the reference's visiting order).
struct alignas(16) TriRecord {
  float v0x, v0y, v0z, e1x;
  float e1y, e1z, e2x, e2y;
  float e2z;
  uint32_t prim;
  uint32_t leaf;
  uint32_t lane;
};
static_assert(sizeof(TriRecord) == 48, "triangle record must be 48 bytes");

// Binary node record for tie resolution: lo3 + parent, hi3 + depth.
struct alignas(16) TieNode {
  float lox, loy, loz;
  int32_t parent;
  float hix, hiy, hiz;
  int32_t depth;
};

struct SceneGeometry {
  std::vector<HostPrim> prims;        // accelerator order (RayQueryHit::primitive_index)
  std::vector<float> boxes;           // 6 floats per prim: lo3, hi3 (padded by 1e-4)
  std::vector<uint32_t> inst_first, inst_count;   // per instance: its flattened primitives
};

struct WideBvh {
  std::vector<WideNode> nodes;
  std::vector<TriRecord> tris;
  std::vector<TieNode> tie_nodes;
  uint32_t binary_nodes = 0;
  uint32_t binary_leaves = 0;
  uint32_t depth = 0;
  uint32_t stack_required = 0;
  bool reference_topology = true;   // traversal tree == reference tree
};

// Dynamic-transform instances: local geometry and per-instance transforms
// (all null when the scene has none).
struct InstanceGeometry {
  const uint32_t* instance_local = nullptr;       // 5 per instance: flags, local first/count vertex, first/count index
  const float* instance_transforms = nullptr;     // 10 per instance: translation3, quaternion xyzw, scale3
  const float* local_vertices = nullptr;
  uint32_t local_vertex_count = 0;
  const uint32_t* local_indices = nullptr;
  uint32_t local_index_count = 0;
};

// A world-space vertex of a dynamic instance: scale, normalized-quaternion
// rotation, translation (transform_instance_vertex and rotate_quat,
// src/pathtracer/CpuBvhAccelerator.cpp:47-74).
void TransformInstanceVertex(const float* local, const float* transform, float out[3]);

// Flattens instances x triangles in the accelerator's order, skipping
// triangles with out-of-range indices (src/pathtracer/CpuBvhAccelerator.cpp:173-247).
bool FlattenScene(const float* vertices, uint32_t vertex_count, const uint32_t* indices,
                  uint32_t index_count, const uint32_t* instances, uint32_t instance_count,
                  SceneGeometry& out, std::string& error, const InstanceGeometry* dyn = nullptr);

// Binary BVH: widest-centroid-axis midpoint split, stable partition,
// count/2 fallback, leaves of <= leaf_threshold primitives, child ids
// allocated pairwise in recursion order (src/cpu/ParallelBvhBuilder.cpp:61-257).
void BuildBinaryBvh(const SceneGeometry& geo, uint32_t leaf_threshold, std::vector<BinNode>& nodes,
                    std::vector<uint32_t>& prim_indices);

// Binned-SAH binary BVH over the same padded primitive boxes (32 bins per
// axis, leaves of <= max_leaf primitives).  Used only as the traversal tree:
// hit ids stay the reference's because ties and the parallel-axis rule are
// resolved against the reference tree (see CollapseToWide).
void BuildSahBvh(const SceneGeometry& geo, uint32_t max_leaf, std::vector<BinNode>& nodes,
                 std::vector<uint32_t>& prim_indices);

// Validates an externally supplied binary BVH against the primitive count.
bool ValidateBinaryBvh(const std::vector<BinNode>& nodes, const std::vector<uint32_t>& prim_indices,
                       size_t prim_count, std::string& error);

// Collapses a binary traversal tree into the wide layout.  Each wide child
// slot is a binary node with its bounds (SetWideSlot).  The leaves of the
// reference's tree stay whole; in another tree subtrees of up to eight triangles
// may become one leaf (CollapseNode).  Triangle records and tie nodes come from the REFERENCE tree
// (ref_nodes / ref_prims): each triangle carries its reference leaf and lane,
// so exact-distance ties and the parallel-axis rule follow the reference even
// when the traversal tree is a different one.
void CollapseToWide(const SceneGeometry& geo, const std::vector<BinNode>& nodes,
                    const std::vector<uint32_t>& prim_indices, const std::vector<BinNode>& ref_nodes,
                    const std::vector<uint32_t>& ref_prims, WideBvh& out);

}  // namespace vkptc
