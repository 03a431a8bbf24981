// traverse.cuh -- wide-BVH closest-hit and any-hit traversal for sm_100a.
//
// Semantics are those of the reference accelerator
// (src/pathtracer/CpuBvhAccelerator.cpp:113-154, 360-477) and its leaf test
// (src/cpu/BvhTriangleIntersector.cpp:25-74):
//  * Moller-Trumbore with |det| < 1e-4 rejected, no backface culling, a hit
//    accepted when 1e-4 < t < best; evaluated in the reference's exact
//    operation order without fused multiply-adds, so t is bit-identical.
//  * Boxes only cull.  Every triangle box is padded by 1e-4 as in the reference.
//    The node test below places a slab within about 2^-24 (|o| + |lo - o|) of
//    where it is, which the padding covers for coordinates of a few hundred, so
//    the box of a triangle that a ray meets is not missed there.  (A triangle
//    whose distance is badly conditioned, |det| near 1e-4, can report one
//    outside its box; whether it is visited, and whether a bound on the distance
//    culls its box, then depends on rounding.)
//  * The reference treats an axis with |d| <= 1e-4 as "parallel" and there only
//    checks that the origin lies inside the slab, which decides which triangles
//    it can test at all.  In its own tree the node test does the same.  In another
//    tree it does not, and leaf_rule_ok() applies the rule to a found hit: it is
//    monotone under box inclusion, so the box of the triangle's leaf in the
//    reference's tree decides it.
//  * Exact distance ties: the reference keeps the first triangle it visits
//    (strict t < best), i.e. the earlier lane of one leaf, or for two leaves
//    the one under the nearer child of their lowest common binary ancestor
//    (left first when the entry distances are equal), since it traverses the
//    binary tree depth first, near child first.  tie_candidate_wins()
//    evaluates exactly that order from the binary tree kept beside the wide one.
//
// The traversal is bound by issued instructions under divergence (about ten of
// a warp's lanes are active per instruction) and by L1 (at 76-80 % of its
// throughput), not by memory bandwidth, so a step is kept short:
//  * A wide node holds its children's boxes as lo[4], hi[4] per axis.  On an
//    axis, with i = 1/d, the slab distances are lo*i - o*i and hi*i - o*i; the
//    sign of d says which is the nearer one, so the node test loads the near
//    and the far four from addresses that depend on it and needs no minimum or
//    maximum per slab: twelve packed multiply-adds (f32x2, two children an
//    instruction), where corner bounds in any order took 24 scalar multiply-adds
//    and 24 min/max, which run at half rate.
//  * The children are ordered by three compare-exchanges: the nearest is exact,
//    the rest are pushed as they come.  A full sort (five) measured 1-3 % slower.
//  * A leaf is its own cursor: the leaf reference of the triangles not yet
//    tested, so no range is kept beside it.
//  * The best hit is kept as its triangle record's index; primitive id, leaf
//    and lane are read from the record when they are needed.
// Against boxes as centre and half extent (three 256-bit loads, 24 packed
// instructions): closest hits of 8,388,608 rays on the 1,046,904-triangle sphere
// 1,459 -> 1,434 us, the 64-job batch 513.6 -> 511.2 ms, a full-HD frame of the
// 2,064,386-triangle grid 19.2 -> 19.8 ms, of the closed box 1.085 -> 1.107 (more
// load instructions).  Those place a slab within 2^-24 (|o| + 3 |c - o|) only: of
// rays aimed at a sphere's vertices from 20 radii away 477 and 996 hits of 60,000
// (reference and SAH tree) differed from the reference's, 344 and 826 now, and
// a ray along a box face beyond coordinates of 1024 could miss the surface in it.
// Three 256-bit loads with the planes swapped by selects: 1,525 us, 527 ms, 19.7 ms.
#pragma once

#include "bvh_layout.h"
#include "common.cuh"

namespace vkptc {

#define kInf __int_as_float(0x7f800000)

// ------------------------------------------------------------ packed floats
// Two floats in one register pair, and the f32x2 multiply-add on them (each lane
// rounded to nearest as the scalar operation is).
typedef unsigned long long F2;
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// 128-bit read-only load of two pairs.
__device__ __forceinline__ void ldg_pairs(const char* p, F2& a, F2& b) {
  asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p));
}

// ------------------------------------------------------------ the ray
// Box-test constants, each twice: 1/d and -o/d per axis.  An axis with
// |d| <= box_eps asks whether the origin lies in the slab, by the reference's rule:
// its 1/d is 2^66, a power of two, so that 2^66 (lo - o) and 2^66 (hi - o) have the
// right signs (on an upper face the far distance is 0: SetWideSlot).  box_eps is
// the reference's 1e-4 where the nodes are the reference's own, 1e-20 (components
// of 0) in other trees, whose boxes can be smaller than the reference's leaves.
struct BoxRay {
  F2 ix, iy, iz, nx, ny, nz;
  uint32_t signs;   // byte k: 16 where axis k's d is negative (its near plane is hi)
};
struct RayPrep {
  float ox, oy, oz, dx, dy, dz;
  BoxRay b;
};

__device__ __forceinline__ void box_axis(float o, float d, float box_eps, uint32_t axis, F2& i2, F2& n2, uint32_t& signs) {
  const float i = fabsf(d) > box_eps ? __frcp_rn(d) : 0x1p66f, n = -(o * i);
  i2 = pack2(i, i);
  n2 = pack2(n, n);
  signs |= i < 0.0f ? 16u << (8u * axis) : 0u;
}

__device__ __forceinline__ RayPrep prep_ray(V3 o, V3 d, float box_eps) {
  RayPrep r;
  r.ox = o.x; r.oy = o.y; r.oz = o.z;
  r.dx = d.x; r.dy = d.y; r.dz = d.z;
  r.b.signs = 0u;
  box_axis(o.x, d.x, box_eps, 0u, r.b.ix, r.b.nx, r.b.signs);
  box_axis(o.y, d.y, box_eps, 1u, r.b.iy, r.b.ny, r.b.signs);
  box_axis(o.z, d.z, box_eps, 2u, r.b.iz, r.b.nz, r.b.signs);
  return r;
}

// The reference's parallel-axis rule for a hit in reference leaf `leaf`: on an
// axis with |d| <= 1e-4 the origin must lie inside that leaf's box.  The
// watertight mode has no such rule: the ray drifts up to 1e-4 t along the axis,
// more than the boxes' padding, so the rule can reject a hit the ray has.
template <bool kWt>
__device__ __forceinline__ bool leaf_rule_ok(const float4* tie, uint32_t leaf, const RayPrep& r) {
  if constexpr (kWt) return true;
  if (fminf(fminf(fabsf(r.dx), fabsf(r.dy)), fabsf(r.dz)) > kEps) return true;
  const float4 a = __ldg(tie + 2 * leaf);
  const float4 b = __ldg(tie + 2 * leaf + 1);
  if (fabsf(r.dx) <= kEps && (r.ox < a.x || r.ox > b.x)) return false;
  if (fabsf(r.dy) <= kEps && (r.oy < a.y || r.oy > b.y)) return false;
  if (fabsf(r.dz) <= kEps && (r.oz < a.z || r.oz > b.z)) return false;
  return true;
}

// Axes with |d| at or below this only test whether the origin is inside.
template <bool kWt>
__device__ __forceinline__ float parallel_eps() { return kWt ? 1e-20f : kEps; }

// The reference's slab test verbatim (no fusion, its own division); returns
// the entry distance.  Only ties evaluate it.
__device__ __forceinline__ bool ref_slab(const float lo[3], const float hi[3], const RayPrep& r, float par_eps,
                                         float& tnear) {
  const float o[3] = {r.ox, r.oy, r.oz};
  const float d[3] = {r.dx, r.dy, r.dz};
  float t_min = kEps, t_max = kInf;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (fabsf(d[a]) <= par_eps) {
      if (o[a] < lo[a] || o[a] > hi[a]) return false;
      continue;
    }
    const float iv = __fdiv_rn(1.0f, d[a]);
    float t0 = __fmul_rn(__fsub_rn(lo[a], o[a]), iv);
    float t1 = __fmul_rn(__fsub_rn(hi[a], o[a]), iv);
    if (t0 > t1) {
      const float tmp = t0;
      t0 = t1;
      t1 = tmp;
    }
    t_min = smax(t_min, t0);
    t_max = smin(t_max, t1);
    if (t_min > t_max) return false;
  }
  tnear = t_min;
  return t_max > kEps;
}

// Moller-Trumbore in the reference's operation order; returns t or -1.
__device__ __forceinline__ float mt_test(const float4 a, const float4 b, const float4 c, const RayPrep& r) {
  const float v0x = a.x, v0y = a.y, v0z = a.z;
  const float e1x = a.w, e1y = b.x, e1z = b.y;
  const float e2x = b.z, e2y = b.w, e2z = c.x;
  const float hx = __fsub_rn(__fmul_rn(r.dy, e2z), __fmul_rn(r.dz, e2y));
  const float hy = __fsub_rn(__fmul_rn(r.dz, e2x), __fmul_rn(r.dx, e2z));
  const float hz = __fsub_rn(__fmul_rn(r.dx, e2y), __fmul_rn(r.dy, e2x));
  const float det = __fadd_rn(__fadd_rn(__fmul_rn(e1x, hx), __fmul_rn(e1y, hy)), __fmul_rn(e1z, hz));
  if (fabsf(det) < kEps) return -1.0f;
  const float inv = __frcp_rn(det);   // correctly rounded, the bits of 1.0f / det
  const float sx = __fsub_rn(r.ox, v0x), sy = __fsub_rn(r.oy, v0y), sz = __fsub_rn(r.oz, v0z);
  const float u = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(sx, hx), __fmul_rn(sy, hy)), __fmul_rn(sz, hz)), inv);
  if (u < 0.0f || u > 1.0f) return -1.0f;
  const float qx = __fsub_rn(__fmul_rn(sy, e1z), __fmul_rn(sz, e1y));
  const float qy = __fsub_rn(__fmul_rn(sz, e1x), __fmul_rn(sx, e1z));
  const float qz = __fsub_rn(__fmul_rn(sx, e1y), __fmul_rn(sy, e1x));
  const float v = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(r.dx, qx), __fmul_rn(r.dy, qy)), __fmul_rn(r.dz, qz)), inv);
  if (v < 0.0f || __fadd_rn(u, v) > 1.0f) return -1.0f;
  const float t = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(e2x, qx), __fmul_rn(e2y, qy)), __fmul_rn(e2z, qz)), inv);
  return t;
}

// Per-ray constants of the watertight test (Woop, Benthin and Wald, "Watertight
// Ray/Triangle Intersection", JCGT 2(1), 2013): kz is the axis of the largest
// |d| (the first on ties), kx and ky follow it cyclically and are swapped when
// d[kz] < 0, which keeps the triangles' winding; the shear maps the ray onto
// +z: sx = d[kx]/d[kz], sy = d[ky]/d[kz], sz = 1/d[kz].
struct WtRay {
  int kx, ky, kz;
  float sx, sy, sz;
};

__device__ __forceinline__ float axis_of(float x, float y, float z, int k) { return k == 0 ? x : (k == 1 ? y : z); }

__device__ __forceinline__ WtRay prep_wt(const RayPrep& r) {
  const float ax = fabsf(r.dx), ay = fabsf(r.dy), az = fabsf(r.dz);
  int kz = 0;
  float m = ax;
  if (ay > m) {
    kz = 1;
    m = ay;
  }
  if (az > m) kz = 2;
  int kx = kz == 2 ? 0 : kz + 1;
  int ky = kx == 2 ? 0 : kx + 1;
  const float dz = axis_of(r.dx, r.dy, r.dz, kz);
  if (dz < 0.0f) {
    const int t = kx;
    kx = ky;
    ky = t;
  }
  WtRay w;
  w.kx = kx;
  w.ky = ky;
  w.kz = kz;
  w.sx = __fdiv_rn(axis_of(r.dx, r.dy, r.dz, kx), dz);
  w.sy = __fdiv_rn(axis_of(r.dx, r.dy, r.dz, ky), dz);
  w.sz = __fdiv_rn(1.0f, dz);
  return w;
}

// The watertight test without back-face culling on a record holding the
// vertices (a, b, c) in the slots of (v0, e1, e2).  The three edge functions
// of the sheared 2D triangle are computed from the vertices themselves, so two
// triangles sharing an edge evaluate it identically (up to sign) and no ray
// passes between them; an edge function that rounds to exactly 0 is redone in
// double (the products are exact there).  Returns t = T/det, or -1 on a miss.
__device__ __forceinline__ float wt_test(const float4 p, const float4 q, const float4 s, const RayPrep& r,
                                         const WtRay& w) {
  const float ax = __fsub_rn(p.x, r.ox), ay = __fsub_rn(p.y, r.oy), az = __fsub_rn(p.z, r.oz);
  const float bx = __fsub_rn(p.w, r.ox), by = __fsub_rn(q.x, r.oy), bz = __fsub_rn(q.y, r.oz);
  const float cx = __fsub_rn(q.z, r.ox), cy = __fsub_rn(q.w, r.oy), cz = __fsub_rn(s.x, r.oz);
  const float akz = axis_of(ax, ay, az, w.kz), bkz = axis_of(bx, by, bz, w.kz), ckz = axis_of(cx, cy, cz, w.kz);
  const float Ax = __fsub_rn(axis_of(ax, ay, az, w.kx), __fmul_rn(w.sx, akz));
  const float Ay = __fsub_rn(axis_of(ax, ay, az, w.ky), __fmul_rn(w.sy, akz));
  const float Bx = __fsub_rn(axis_of(bx, by, bz, w.kx), __fmul_rn(w.sx, bkz));
  const float By = __fsub_rn(axis_of(bx, by, bz, w.ky), __fmul_rn(w.sy, bkz));
  const float Cx = __fsub_rn(axis_of(cx, cy, cz, w.kx), __fmul_rn(w.sx, ckz));
  const float Cy = __fsub_rn(axis_of(cx, cy, cz, w.ky), __fmul_rn(w.sy, ckz));
  float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
  float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
  float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
  if (U == 0.0f || V == 0.0f || W == 0.0f) {
    U = __double2float_rn(__dsub_rn(__dmul_rn(Cx, By), __dmul_rn(Cy, Bx)));
    V = __double2float_rn(__dsub_rn(__dmul_rn(Ax, Cy), __dmul_rn(Ay, Cx)));
    W = __double2float_rn(__dsub_rn(__dmul_rn(Bx, Ay), __dmul_rn(By, Ax)));
  }
  if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return -1.0f;
  const float det = __fadd_rn(__fadd_rn(U, V), W);
  if (det == 0.0f) return -1.0f;
  const float Az = __fmul_rn(w.sz, akz), Bz = __fmul_rn(w.sz, bkz), Cz = __fmul_rn(w.sz, ckz);
  const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
  return __fdiv_rn(T, det);
}

// The configured triangle test: the reference's Moller-Trumbore, or watertight.
template <bool kWt>
__device__ __forceinline__ float tri_test(const float4 a, const float4 b, const float4 c, const RayPrep& r,
                                          const WtRay& w) {
  if constexpr (kWt) return wt_test(a, b, c, r, w);
  else return mt_test(a, b, c, r);
}

__device__ __forceinline__ void tie_box(const float4* tie, int32_t id, float lo[3], float hi[3]) {
  const float4 a = __ldg(tie + 2 * id);
  const float4 b = __ldg(tie + 2 * id + 1);
  lo[0] = a.x; lo[1] = a.y; lo[2] = a.z;
  hi[0] = b.x; hi[1] = b.y; hi[2] = b.z;
}
__device__ __forceinline__ int32_t tie_parent(const float4* tie, int32_t id) {
  return __float_as_int(__ldg(tie + 2 * id).w);
}
__device__ __forceinline__ int32_t tie_depth(const float4* tie, int32_t id) {
  return __float_as_int(__ldg(tie + 2 * id + 1).w);
}

// True when the candidate (leaf_b, lane_b) is visited before the incumbent
// (leaf_a, lane_a) by the reference's depth-first near-first traversal.
__device__ __forceinline__ bool tie_candidate_wins(const float4* tie, const RayPrep& r, float par_eps, uint32_t leaf_a,
                                                   uint32_t lane_a, uint32_t leaf_b, uint32_t lane_b) {
  if (leaf_a == leaf_b) return lane_b < lane_a;
  int32_t a = static_cast<int32_t>(leaf_a), b = static_cast<int32_t>(leaf_b);
  int32_t da = tie_depth(tie, a), db = tie_depth(tie, b);
  while (da > db && a > 0) { a = tie_parent(tie, a); --da; }
  while (db > da && b > 0) { b = tie_parent(tie, b); --db; }
  // Climb together to the children of the lowest common ancestor; the root
  // (id 0, parent -1) ends the walk on malformed input.
  while (a > 0 && b > 0 && tie_parent(tie, a) != tie_parent(tie, b)) {
    a = tie_parent(tie, a);
    b = tie_parent(tie, b);
  }
  if (a <= 0 || b <= 0) return false;
  float lo[3], hi[3];
  float ta = 0.0f, tb = 0.0f;
  tie_box(tie, a, lo, hi);
  ref_slab(lo, hi, r, par_eps, ta);
  tie_box(tie, b, lo, hi);
  ref_slab(lo, hi, r, par_eps, tb);
  // Sibling ids are allocated (left, right) consecutively: left is the smaller.
  const bool a_left = a < b;
  const float t_left = a_left ? ta : tb, t_right = a_left ? tb : ta;
  const bool left_first = t_left <= t_right;
  const bool a_first = (a_left == left_first);
  return !a_first;
}

struct TraceStats {
  uint32_t nodes = 0, leaves = 0, tris = 0, rays = 0;
};

// ------------------------------------------------------------ one step
// Entry distances of a wide node's children (infinity: missed, or farther than
// tmax) and their refs.  A NaN bound or ray component passes its axis.
__device__ __forceinline__ void node_test(const float4* np, const BoxRay& b, float tmax, float (&t)[4], int32_t (&c)[4]) {
  const char* p = reinterpret_cast<const char*>(np);
  const uint32_t sx = b.signs & 16u, sy = (b.signs >> 8) & 16u, sz = b.signs >> 16;
  F2 nx[2], ny[2], nz[2], fx[2], fy[2], fz[2];
  ldg_pairs(p + sx, nx[0], nx[1]);
  ldg_pairs(p + (sx ^ 16u), fx[0], fx[1]);
  ldg_pairs(p + 32 + sy, ny[0], ny[1]);
  ldg_pairs(p + 32 + (sy ^ 16u), fy[0], fy[1]);
  ldg_pairs(p + 64 + sz, nz[0], nz[1]);
  ldg_pairs(p + 64 + (sz ^ 16u), fz[0], fz[1]);
  const int4 ch = __ldg(reinterpret_cast<const int4*>(np + 6));
  c[0] = ch.x;
  c[1] = ch.y;
  c[2] = ch.z;
  c[3] = ch.w;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    float ax[2], ay[2], az[2], bx[2], by[2], bz[2];
    unpack2(fma2(nx[k], b.ix, b.nx), ax[0], ax[1]);
    unpack2(fma2(ny[k], b.iy, b.ny), ay[0], ay[1]);
    unpack2(fma2(nz[k], b.iz, b.nz), az[0], az[1]);
    unpack2(fma2(fx[k], b.ix, b.nx), bx[0], bx[1]);
    unpack2(fma2(fy[k], b.iy, b.ny), by[0], by[1]);
    unpack2(fma2(fz[k], b.iz, b.nz), bz[0], bz[1]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int s = 2 * k + e;
      const float tn = fmaxf(fmaxf(fmaxf(ax[e], ay[e]), az[e]), kEps);
      const float tf = fminf(fminf(fminf(bx[e], by[e]), bz[e]), tmax);
      t[s] = tn <= tf && (s == 0 || c[s] != kEmptyChild) ? tn : kInf;   // slot 0 is never empty
    }
  }
}

// Triangle record k (its three words are at 3k).
__device__ __forceinline__ uint32_t leaf_cursor(int32_t ref) { return ~static_cast<uint32_t>(ref); }

// Traversal stack of (ref, entry distance): the first `scap` entries in shared
// memory (interleaved per thread, so consecutive threads hit distinct banks),
// the rest in a per-thread slab in global memory.  The host sizes scap plus the
// slab from the BVH's exact worst case.
struct TwoLevelStack {
  int2* smem;     // this thread's entry 0; entry i at smem[i * sstride]
  int sstride;
  int scap;
  int2* spill;    // this thread's spill entry 0; entry i at spill[i * gstride]
  int gstride;
  int total;      // scap + spill entries
  __device__ __forceinline__ void put(int i, int2 e) const {
    if (i < scap) smem[i * sstride] = e;
    else spill[(i - scap) * gstride] = e;
  }
  __device__ __forceinline__ int2 get(int i) const {
    return i < scap ? smem[i * sstride] : spill[(i - scap) * gstride];
  }
};
// A stack held whole in shared memory.
__device__ __forceinline__ TwoLevelStack smem_stack_of(int2* base, int stride, int cap) {
  return TwoLevelStack{base, stride, cap, nullptr, 0, cap};
}

// Geometry a query traverses (one launch may serve several scenes).
struct GeoView {
  const float4* nodes;
  const float4* tris;
  const float4* tie;
  uint32_t prim_count;
  float box_eps;   // |d| up to which an axis of the node test uses the inside rule
};

__host__ __device__ __forceinline__ GeoView geo_of(const DevScene& s) {
  return GeoView{s.nodes, s.tris, s.tie, s.prim_count, s.box_eps};
}

// What a kernel's queries ask for: the closest hit, any hit, or a mixture that
// the source decides per query (Src::any(j)).
constexpr int kQueryClosest = 0, kQueryAny = 1, kQueryMixed = 2;

struct LaneState {
  RayPrep r;
  WtRay w;          // watertight test constants (unused by the Moller-Trumbore kernels)
  float t;          // closest: best distance so far; any: the query's upper bound
  int32_t best;     // closest: triangle record of the best hit; any: 0 when occluded; -1: none
  int32_t ref;      // >= 0: wide node to visit; < 0: leaf, from its next triangle on
  int sp;
  bool any;         // kQueryMixed: this query ends at its first hit
};

// tmax: hits at or beyond it do not count (infinity: no bound).
template <bool kWt>
__device__ __forceinline__ void lane_begin(LaneState& L, V3 o, V3 d, float tmax, float box_eps) {
  L.r = prep_ray(o, d, box_eps);
  if constexpr (kWt) L.w = prep_wt(L.r);
  L.t = tmax;
  L.best = -1;
  L.ref = 0;
  L.sp = 0;
}

template <bool kStats>
__device__ __forceinline__ void lane_enter(LaneState& L, int32_t ref, TraceStats& st) {
  L.ref = ref;
  if (kStats && ref < 0) {
    ++st.leaves;
    st.tris += (leaf_cursor(ref) & 7u) + 1u;
  }
}

// One step of a query: one wide node or one triangle.  A warp's lanes diverge
// between the two at every step; with whole leaves per step a lane in a leaf
// would hold the warp for several triangle tests, with single triangles the two
// branches cost about the same.  Letting the warp vote for one of the two
// branches per step gained 10 % on camera rays of a sparse scene and lost as
// much on others.  tie() returns the scene's tie records.  Returns true when
// the query has finished.
template <int kMode, bool kStats, bool kWt, class TieFn>
__device__ __forceinline__ bool lane_step(LaneState& L, const float4* nodes, const float4* tris, const TieFn& tie,
                                          const TwoLevelStack& stk, TraceStats& st, uint32_t& err) {
  if (L.ref < 0) {
    const uint32_t u = leaf_cursor(L.ref);   // (first triangle << 3) | (triangles left - 1)
    const float4* tp = tris + 3u * (u >> 3);
    const float4 a = __ldg(tp), b = __ldg(tp + 1), cc = __ldg(tp + 2);
    const float th = tri_test<kWt>(a, b, cc, L.r, L.w);
    if (th > kEps && (kMode == kQueryAny ? th < L.t : th <= L.t) &&
        leaf_rule_ok<kWt>(tie(), __float_as_uint(cc.z), L.r)) {
      if (kMode == kQueryAny) {
        L.best = 0;
        return true;
      }
      bool take = th < L.t;
      if (!take && L.best >= 0) {   // L.best < 0: th is the query's bound, which is no hit
        const float4 ic = __ldg(tris + 3u * static_cast<uint32_t>(L.best) + 2);
        take = tie_candidate_wins(tie(), L.r, parallel_eps<kWt>(), __float_as_uint(ic.z), __float_as_uint(ic.w),
                                  __float_as_uint(cc.z), __float_as_uint(cc.w));
      }
      if (take) {
        L.t = th;
        L.best = static_cast<int32_t>(u >> 3);
        if (kMode == kQueryMixed && L.any) return true;
      }
    }
    if (u & 7u) {
      L.ref = ~static_cast<int32_t>(u + 7u);   // the next triangle, one fewer left
      return false;
    }
  } else {
    float t[4];
    int32_t c[4];
    if (kStats) ++st.nodes;
    node_test(nodes + 8ll * L.ref, L.r.b, L.t, t, c);
#define VKPTC_CSWAP(i, j)                                             \
  {                                                                   \
    const bool sw = t[j] < t[i];                                      \
    const float tn = sw ? t[j] : t[i], tx = sw ? t[i] : t[j];         \
    const int32_t cn = sw ? c[j] : c[i], cx = sw ? c[i] : c[j];       \
    t[i] = tn; t[j] = tx; c[i] = cn; c[j] = cx;                       \
  }
    VKPTC_CSWAP(0, 1) VKPTC_CSWAP(2, 3) VKPTC_CSWAP(0, 2)
#undef VKPTC_CSWAP
    if (t[0] < kInf) {
      if (L.sp + 3 <= stk.scap) {
        int2* p = stk.smem + L.sp * stk.sstride;
        if (t[3] < kInf) {
          *p = make_int2(c[3], __float_as_int(t[3]));
          p += stk.sstride;
          ++L.sp;
        }
        if (t[1] < kInf) {
          *p = make_int2(c[1], __float_as_int(t[1]));
          p += stk.sstride;
          ++L.sp;
        }
        if (t[2] < kInf) {
          *p = make_int2(c[2], __float_as_int(t[2]));
          ++L.sp;
        }
      } else {
        const int order[3] = {3, 1, 2};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (!(t[order[k]] < kInf)) continue;
          if (L.sp < stk.total) {
            stk.put(L.sp, make_int2(c[order[k]], __float_as_int(t[order[k]])));
            ++L.sp;
          } else {
            err = 1u;
          }
        }
      }
      lane_enter<kStats>(L, c[0], st);
      return false;
    }
  }
  // Pop the next entry that can still hold a hit no farther than the best.
  while (L.sp > 0) {
    --L.sp;
    const int2 e = stk.get(L.sp);
    if (kMode == kQueryAny || __int_as_float(e.y) <= L.t) {
      lane_enter<kStats>(L, e.x, st);
      return false;
    }
  }
  return true;
}

// ------------------------------------------------------------ one query per thread
// Closest hit.  best_t = +inf and prim = kMiss on a miss.  `err` receives 1 on
// a stack overflow (which the host-side sizing rules out).
template <bool kStats, bool kWt = false>
__device__ __forceinline__ void trace_closest(const DevScene& s, V3 o, V3 d, const TwoLevelStack& stk, float& best_t,
                                              uint32_t& best_prim, TraceStats& st, uint32_t& err) {
  best_t = kInf;
  best_prim = kMiss;
  if (s.prim_count == 0u) return;
  LaneState L;
  lane_begin<kWt>(L, o, d, kInf, s.box_eps);
  const auto tie = [&]() { return s.tie; };
  while (!lane_step<kQueryClosest, kStats, kWt>(L, s.nodes, s.tris, tie, stk, st, err)) {
  }
  best_t = L.t;
  if (L.best >= 0) best_prim = __float_as_uint(__ldg(s.tris + 3u * static_cast<uint32_t>(L.best) + 2).y);
}

// Any hit with 1e-4 < t < tmax.  Returns true when occluded.
template <bool kStats, bool kWt = false>
__device__ __forceinline__ bool trace_any(const DevScene& s, V3 o, V3 d, float tmax, const TwoLevelStack& stk,
                                          TraceStats& st, uint32_t& err) {
  if (s.prim_count == 0u || !(tmax > kEps)) return false;
  LaneState L;
  lane_begin<kWt>(L, o, d, tmax, s.box_eps);
  const auto tie = [&]() { return s.tie; };
  while (!lane_step<kQueryAny, kStats, kWt>(L, s.nodes, s.tris, tie, stk, st, err)) {
  }
  return L.best >= 0;
}

// ------------------------------------------------------------ persistent
// Persistent traversal over `n` queries supplied by Src:
//   Src::load(j, o, d, tmax, geo) and Src::finish(j, t, prim) (any-hit: prim = occluded);
//   Src::kUniform: one scene serves the whole launch (its pointers then stay in
//   uniform registers), and Src::geo_at(j): query j's scene, for the rare reads
//   of the tie records.
// kQueryMixed: Src::any(j) says whether query j ends at its first hit, and
// Src::finish(j, t, prim, o, d, tmax) may return true to go on with a new
// origin and bound (o and tmax updated) as the same query; with kStats,
// Src::traced(j) whether it counts as a ray.
// Each warp keeps its lanes busy: whenever lanes are idle it claims that many
// query ids with one atomic (warp-aggregated) and refills them.  `steps`
// packs two limits: the low 16 bits are the most traversal steps between
// refills; the high bits, when non-zero, a refill threshold -- the warp
// leaves the step loop for a refill as soon as that many lanes are idle
// (checked after every step).  Without a threshold the lanes run the full
// number of steps between refills.  At most one query per thread of the launch:
// no counter is needed (fetch may be null); the queries are spread evenly over
// all warps, because a warp takes as long as its lanes' divergent steps together
// (1,000 rays on the 130k-triangle field, queries and clearing of the counter:
// 46 us in full warps with the counter, 38 us in full warps without, 18.5 us
// spread).  st: the work of closest-hit queries, st_any
// that of any-hit queries (the same object where a launch has one kind).
template <class Src, int kMode, bool kStats, bool kWt = false>
__device__ __forceinline__ void persistent_traverse(const Src& src, uint32_t n, uint32_t* fetch, TwoLevelStack stk,
                                                    int steps, TraceStats& st, TraceStats& st_any, uint32_t& err) {
  const unsigned lane_id = threadIdx.x & 31u;
  const int max_steps = steps & 0xFFFF;
  const int refill_min = steps >> 16;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const bool spread = n <= 32u * warps;
  LaneState L;
  const float4* nodes = nullptr;
  const float4* tris = nullptr;
  if constexpr (Src::kUniform) {
    nodes = src.geo.nodes;
    tris = src.geo.tris;
  }
  bool active = false;
  bool exhausted = false;
  uint32_t tag = 0u;
  const auto tie = [&]() { return src.geo_at(tag).tie; };
  // The end of query j: its result stored, or (mixed) the lane restarted.
  // Returns true when the query goes on.
  const auto finish = [&](uint32_t j, LaneState& l) {
    const bool any = kMode == kQueryAny || (kMode == kQueryMixed && l.any);
    uint32_t prim = any ? 0u : kMiss;
    if (l.best >= 0) prim = any ? 1u : __float_as_uint(__ldg(tris + 3u * static_cast<uint32_t>(l.best) + 2).y);
    if constexpr (kMode == kQueryMixed) {
      V3 o = mk(l.r.ox, l.r.oy, l.r.oz);
      const V3 d = mk(l.r.dx, l.r.dy, l.r.dz);
      float tmax;
      if (src.finish(j, l.t, prim, o, d, tmax)) {
        lane_begin<kWt>(l, o, d, tmax, src.geo_at(j).box_eps);
        return true;
      }
    } else {
      src.finish(j, l.t, prim);
    }
    if constexpr (kStats && kMode == kQueryMixed) {
      if (!src.traced(j)) return false;
    }
    if (kStats) ++(any ? st_any : st).rays;
    return false;
  };
  const auto step = [&](LaneState& l) {
    if constexpr (kStats && kMode == kQueryMixed) {
      if (src.shadow(tag)) return lane_step<kMode, kStats, kWt>(l, nodes, tris, tie, stk, st_any, err);
    }
    return lane_step<kMode, kStats, kWt>(l, nodes, tris, tie, stk, st, err);
  };
  while (true) {
    const unsigned idle = __ballot_sync(0xffffffffu, !active);
    if (idle != 0u && !exhausted) {
      uint32_t base = 0u, limit = n;
      if (!spread) {
        if (lane_id == 0u) base = atomicAdd(fetch, static_cast<uint32_t>(__popc(idle)));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) exhausted = true;
      } else {
        const uint32_t share = (n + warps - 1u) / warps;
        base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * share;
        limit = min(n, base + share);
        exhausted = true;
      }
      if (!active) {
        const uint32_t j = base + static_cast<uint32_t>(__popc(idle & ((1u << lane_id) - 1u)));
        if (j < limit && j >= base) {
          V3 o, d;
          float tmax;
          GeoView g;
          src.load(j, o, d, tmax, g);
          if constexpr (!Src::kUniform) {
            nodes = g.nodes;
            tris = g.tris;
          }
          if constexpr (kMode == kQueryMixed) L.any = src.any(j);
          lane_begin<kWt>(L, o, d, kMode == kQueryClosest ? kInf : tmax, g.box_eps);
          if (g.prim_count == 0u || (kMode != kQueryClosest && !(tmax > kEps))) {
            finish(j, L);
          } else {
            tag = j;
            active = true;
          }
        }
      }
    }
    if (!__any_sync(0xffffffffu, active)) {
      if (exhausted) break;
      continue;   // every query claimed ended at load: there may be more
    }
    if (refill_min == 0) {
      if (active) {
        for (int k = 0; k < max_steps; ++k) {
          if (step(L) && !finish(tag, L)) {
            active = false;
            break;
          }
        }
      }
    } else {
      for (int k = 0; k < max_steps; ++k) {
        if (active && step(L) && !finish(tag, L)) active = false;
        const unsigned idle_now = __ballot_sync(0xffffffffu, !active);
        if (idle_now == 0xffffffffu || (!exhausted && __popc(idle_now) >= refill_min)) break;
      }
    }
  }
}

}  // namespace vkptc
