// kernels.cu -- wavefront path tracing and ray-query kernels (sm_100a).
//
// The integrator restates the reference's scalar CPU tracer:
//   camera_rays / shade_pixel   src/pathtracer/ScalarCpuPathTracer.Render.cpp:55-119, 228-284
//   trace                       src/pathtracer/ScalarCpuPathTracer.cpp:1148-1289
//   sample_direct_light         src/pathtracer/ScalarCpuPathTracer.cpp:1022-1118
//   light_pdf / MisWeight       src/pathtracer/ScalarCpuPathTracer.cpp:1120-1146
//   hemisphere / Phong lobe     src/pathtracer/ScalarCpuPathTracer.cpp:978-1020
//   FilmBuffer add / resolve    src/pathtracer/FilmBuffer.cpp:80-91, 160-214
// split into wavefront stages that exchange structure-of-arrays queues:
//   raygen -> for each depth: trace (closest hits of this depth's paths and the
//   previous depth's shadow queries, one launch) -> shade (material, NEE set-up,
//   BSDF sample, Russian roulette; appends shadow queries and the next extension
//   queue with warp-aggregated atomics) -> accumulate into the film in sample
//   order.  Scenes with SDF primitives add two load-balanced stages (below).
// The per-path RNG stream is keyed exactly as the reference keys it, so the
// wavefront reordering does not change any random number a path draws, and
// the stages add radiance terms in the reference's order (emission, then the
// NEE term of the same bounce, then the next bounce).
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "integrator.cuh"
#include "traverse.cuh"

namespace vkptc {

size_t StackSmemBytes(int block, int cap) { return static_cast<size_t>(block) * cap * sizeof(int2); }

size_t SpillEntries(const LaunchShape& ls) {
  const int extra = ls.stack_cap - ls.smem_entries;
  return extra > 0 ? static_cast<size_t>(ls.grid) * ls.block * extra : 0u;
}

// ============================================================ query sources
// Each source supplies queries to persistent_traverse() and consumes results.
struct RaysSource {   // batched ray queries from a ray array
  GeoView geo;
  static constexpr bool kUniform = true;
  __device__ __forceinline__ const GeoView& geo_at(uint32_t) const { return geo; }
  const float* rays;
  const float* tmax;
  uint32_t* prim_out;
  float* t_out;
  bool any;
  __device__ __forceinline__ void load(uint32_t j, V3& o, V3& d, float& tm, GeoView& g) const {
    g = geo;
    const float2* rp = reinterpret_cast<const float2*>(rays + 6ull * j);
    const float2 a = __ldg(rp), b = __ldg(rp + 1), c = __ldg(rp + 2);
    o = mk(a.x, a.y, b.x);
    d = mk(b.y, c.x, c.y);
    tm = tmax ? __ldg(tmax + j) : kInf;
  }
  __device__ __forceinline__ void finish(uint32_t j, float t, uint32_t prim) const {
    prim_out[j] = prim;
    if (t_out) t_out[j] = any ? (prim ? 0.0f : kInf) : t;
  }
};

// A wave's traversal queries: the extension rays of the queued paths (closest
// hit), then the shadow queries of the previous depth's shading (its term is
// added when visible).  A shadow query is any-hit; with kTrans (the scene has
// transmissive materials) it is the reference's closest-hit loop that steps
// through up to 8 transmissive occluders
// (src/pathtracer/ScalarCpuPathTracer.cpp:1067-1087), bounded by the distance
// that is left, and goes on in the same lane after each of them.
constexpr uint32_t kDroppedQuery = 0xFFFFFFFFu;   // sh_path of a query an SDF occludes

template <bool kTrans>
struct WaveTraceSource {
  GeoView geo;
  const uint32_t* q;
  const float4* ray_o;
  const float4* ray_d;
  float2* hit;
  float4* sh_o;         // kTrans rewrites origin's w (the distance left)
  float4* sh_d;         // and direction's w (occluders passed, bits)
  const float4* sh_c;
  const uint32_t* sh_path;
  float4* rad;
  uint32_t n_ext;
  const float4* shade;
  const float* materials;
  uint32_t material_count;
  static constexpr bool kUniform = true;
  __device__ __forceinline__ const GeoView& geo_at(uint32_t) const { return geo; }
  __device__ __forceinline__ bool shadow(uint32_t j) const { return j >= n_ext; }
  __device__ __forceinline__ bool any(uint32_t j) const { return !kTrans && j >= n_ext; }
  // A query that an SDF primitive occludes is no traversal ray.
  __device__ __forceinline__ bool traced(uint32_t j) const { return j < n_ext || sh_path[j - n_ext] != kDroppedQuery; }
  __device__ __forceinline__ void load(uint32_t j, V3& o, V3& d, float& tm, GeoView& g) const {
    g = geo;
    const bool sh = j >= n_ext;
    const uint32_t k = sh ? j - n_ext : q[j];
    const float4 a = (sh ? sh_o : ray_o)[k], b = (sh ? sh_d : ray_d)[k];
    o = mk(a.x, a.y, a.z);
    d = mk(b.x, b.y, b.z);
    tm = sh ? a.w : kInf;
  }
  // Returns true when the query goes on from a new origin.
  __device__ __forceinline__ bool finish(uint32_t j, float t, uint32_t prim, V3& o, V3 d, float& tmax) const {
    if (j < n_ext) {
      hit[q[j]] = make_float2(t, __uint_as_float(prim));
      return false;
    }
    const uint32_t k = j - n_ext;
    if constexpr (kTrans) {
      if (prim != kMiss) {
        const uint32_t mat_index = __float_as_uint(__ldg(shade + prim).w);
        const uint32_t mi = mat_index < material_count - 1u ? mat_index : material_count - 1u;
        const float* mm = materials + 16u * mi;
        if (!(static_cast<uint32_t>(mm[7] + 0.5f) == 5u || mm[10] > 0.05f)) return false;   // occluded
        const float adv = t + 0.004f;
        const float left = sh_o[k].w - adv;
        const uint32_t passed = __float_as_uint(sh_d[k].w) + 1u;
        if (passed < 8u && left > 0.004f) {
          o = add(o, mul(d, adv));
          tmax = left;
          sh_o[k].w = left;
          sh_d[k].w = __uint_as_float(passed);
          return true;
        }
      }
    } else {
      if (prim) return false;
    }
    const uint32_t path = sh_path[k];
    if (path == kDroppedQuery) return false;
    const float4 c = sh_c[k];
    float4 r = rad[path];
    r.x = r.x + c.x;
    r.y = r.y + c.y;
    r.z = r.z + c.z;
    rad[path] = r;
    return false;
  }
};

// SDF closest hits of the extension queue, folded into the triangle hits.
struct WaveSdfExtSource {
  const float4* sdf;
  uint32_t sdf_count;
  const uint32_t* q;
  const float4* ray_o;
  const float4* ray_d;
  float2* hit;
  __device__ __forceinline__ void load(uint32_t j, SdfLane& L) const {
    L.sdf = sdf;
    L.count = sdf_count;
    const uint32_t p = q[j];
    const float4 a = ray_o[p], b = ray_d[p];
    const float2 h = hit[p];
    L.o = mk(a.x, a.y, a.z);
    L.d = mk(b.x, b.y, b.z);
    L.best = h.x;
    L.prim = __float_as_uint(h.y);
  }
  __device__ __forceinline__ void finish(uint32_t j, const SdfLane& L) const {
    hit[q[j]] = make_float2(L.best, __uint_as_float(L.prim));
  }
};

// SDF occlusion of the shadow queries: an occluded query is dropped (its bound
// set to 0, so the triangle any-hit does no work for it either).
struct WaveSdfShadowSource {
  const float4* sdf;
  uint32_t sdf_count;
  float4* sh_o;
  const float4* sh_d;
  uint32_t* sh_path;
  __device__ __forceinline__ void load(uint32_t k, SdfLane& L) const {
    L.sdf = sdf;
    L.count = sdf_count;
    const float4 a = sh_o[k], b = sh_d[k];
    L.o = mk(a.x, a.y, a.z);
    L.d = mk(b.x, b.y, b.z);
    L.best = a.w;
    L.prim = 0u;
  }
  __device__ __forceinline__ void finish(uint32_t k, const SdfLane& L) const {
    if (L.prim == 0u) return;
    sh_path[k] = kDroppedQuery;
    sh_o[k].w = 0.0f;
  }
};

__device__ __forceinline__ TwoLevelStack launch_stack(int2* smem_stack, int scap, int2* spill, int total) {
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  return TwoLevelStack{smem_stack + threadIdx.x, static_cast<int>(blockDim.x), scap, spill ? spill + gtid : nullptr,
                       static_cast<int>(gridDim.x * blockDim.x), total};
}

// The traversal kernels run at 64 registers (at least 1024 threads per SM):
// they wait on node and triangle loads more than on anything else, and at 74
// registers (24 warps per SM instead of 32) a full-HD frame of the 2M-triangle
// grid took 37.2 ms instead of 30.7.
// =============================================================== ray queries
template <bool kAny, bool kStats, bool kWt>
__global__ void __launch_bounds__(256, 4) k_trace_rays(DevScene s, RaysSource src, uint32_t n, uint32_t* fetch,
                                                       int scap, int2* spill, int total, int steps, DevCounters* ctr,
                                                       uint32_t* err) {
  extern __shared__ int2 smem_stack[];
  TraceStats st;
  uint32_t lerr = 0u;
  persistent_traverse<RaysSource, kAny ? kQueryAny : kQueryClosest, kStats, kWt>(
      src, n, fetch, launch_stack(smem_stack, scap, spill, total), steps, st, st, lerr);
  if (kStats) {
    warp_count(&ctr->nodes, st.nodes);
    warp_count(&ctr->leaves, st.leaves);
    warp_count(&ctr->tris, st.tris);
    warp_count(&ctr->ext_rays, st.rays);
  }
  if (lerr) atomicOr(err, lerr);
}

cudaError_t LaunchTraceRays(const DevScene& s, const float* rays, const float* tmax, uint64_t n, bool any_hit,
                            uint32_t* prim_out, float* t_out, const LaunchShape& ls, DevCounters* ctr,
                            uint32_t* err, uint32_t* fetch) {
  if (n == 0) return cudaSuccess;
  const size_t smem = StackSmemBytes(ls.block, ls.smem_entries);
  const RaysSource src{geo_of(s), rays, tmax, prim_out, t_out, any_hit};
  const uint32_t n32 = static_cast<uint32_t>(n);
  // At most one ray per resident thread: the kernel spreads them over its warps
  // without the query counter, so there is none to clear, and warps that would
  // get nothing are not launched.
  const uint32_t per_block = static_cast<uint32_t>(ls.block) / 32u;
  uint32_t grid = static_cast<uint32_t>(ls.grid);
  if (n <= 32ull * grid * per_block) {
    const uint32_t share = (n32 + grid * per_block - 1u) / (grid * per_block);
    grid = ((n32 + share - 1u) / share + per_block - 1u) / per_block;
  } else {
    const cudaError_t e = cudaMemsetAsync(fetch, 0, sizeof(uint32_t), ls.stream);
    if (e != cudaSuccess) return e;
  }
#define VKPTC_TR(A, S, W) \
  k_trace_rays<A, S, W><<<grid, ls.block, smem, ls.stream>>>(s, src, n32, fetch, ls.smem_entries, ls.spill, ls.stack_cap, ls.steps, ctr, err)
#define VKPTC_TR2(A, S) \
  if (s.watertight) VKPTC_TR(A, S, true); \
  else VKPTC_TR(A, S, false)
  if (any_hit) {
    if (ctr) VKPTC_TR2(true, true);
    else VKPTC_TR2(true, false);
  } else {
    if (ctr) VKPTC_TR2(false, true);
    else VKPTC_TR2(false, false);
  }
#undef VKPTC_TR2
#undef VKPTC_TR
  return cudaGetLastError();
}

// Control words of a wave (WaveState::counts).
constexpr int kWaveExt = 0;           // extension queue sizes: words 0, 1
constexpr int kWaveShadow = 2;        // shadow queue size by the depth that fills it (even, odd): words 2, 3
constexpr int kWaveFetch = 4;         // query counters of the trace stage; word 5: its shadow part alone
constexpr int kWaveFetchSdf = 6, kWaveFetchSdfShadow = 7;

// ==================================================================== raygen
// Slots of a wave: the tile's pixels in 8x4 tiles, 32 pixels at a time, all
// samples of 32 pixels before the next, so that neighbouring warps' paths start
// in the same place (the slots of the last, incomplete 32 are sample-major).
__device__ __forceinline__ uint32_t wave_slot(uint32_t k, uint32_t sl, uint32_t tile_px, uint32_t samples) {
  const uint32_t full = tile_px & ~31u;
  if (k < full) return (k & ~31u) * samples + sl * 32u + (k & 31u);
  return full * samples + sl * (tile_px - full) + (k - full);
}

template <bool kParity>
__global__ void __launch_bounds__(256) k_raygen(DevScene s, DevSettings st, WaveState w, WaveTile tile) {
  const uint32_t tile_px = tile.w * tile.h;
  const uint32_t n = tile_px * tile.sample_count;
  const uint32_t full = tile_px & ~31u, rest = tile_px - full;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t sl, k;
    if (i < full * tile.sample_count) {
      const uint32_t g = (i >> 5) / tile.sample_count;
      sl = (i >> 5) - g * tile.sample_count;
      k = 32u * g + (i & 31u);
    } else {
      const uint32_t r = i - full * tile.sample_count;
      sl = r / rest;
      k = full + r - sl * rest;
    }
    const uint32_t pl = tile_order_pixel(k, tile.w, tile.h);
    const uint32_t x = tile.x + pl % tile.w, y = tile.y + pl / tile.w;
    V3 o, d;
    uint64_t rng;
    camera_path<kParity>(s, st, x, y, tile.first_sample + sl, o, d, rng);
    w.rng[i] = rng;
    w.ray_o[i] = make_float4(o.x, o.y, o.z, 0.0f);
    w.ray_d[i] = make_float4(d.x, d.y, d.z, 0.0f);
    w.thr[i] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    w.rad[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    w.q[0][i] = i;
  }
  if (blockIdx.x == 0 && threadIdx.x < 8u) ctl_word(w.counts, threadIdx.x) = threadIdx.x == kWaveExt ? n : 0u;
}

// ===================================================================== trace
// The closest hits of depth `depth`'s paths and the shadow queries depth - 1's
// shading left (persistent warps): neither touches what the other reads or
// writes, and one launch has one tail instead of two.  `parts`: 1 the
// extension rays, 2 the shadow queries, 3 both.  Zeroes the next extension
// queue's size and the shadow queue size the coming shading appends to.
template <bool kStats, bool kWt, bool kTrans>
__global__ void __launch_bounds__(256, 4) k_trace(DevScene s, WaveState w, const uint32_t* q, uint32_t depth,
                                                  uint32_t parts, int scap, int2* spill, int total, int steps,
                                                  DevCounters* ctr, uint32_t* err) {
  extern __shared__ int2 smem_stack[];
  const uint32_t cur = depth & 1u;
  const uint32_t n_ext = (parts & 1u) ? ctl_word(w.counts, kWaveExt + cur) : 0u;
  const uint32_t n_sh = (parts & 2u) ? ctl_word(w.counts, kWaveShadow + (cur ^ 1u)) : 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0 && (parts & 1u)) {
    ctl_word(w.counts, kWaveExt + (cur ^ 1u)) = 0u;
    ctl_word(w.counts, kWaveShadow + cur) = 0u;
    ctl_word(w.counts, kWaveFetchSdf) = 0u;
    ctl_word(w.counts, kWaveFetchSdfShadow) = 0u;
  }
  const WaveTraceSource<kTrans> src{geo_of(s), q, w.ray_o, w.ray_d, w.hit, w.sh_o, w.sh_d, w.sh_c, w.sh_path, w.rad,
                                    n_ext, s.shade, s.materials, s.material_count};
  TraceStats st, st_sh;
  uint32_t lerr = 0u;
  persistent_traverse<WaveTraceSource<kTrans>, kQueryMixed, kStats, kWt>(
      src, n_ext + n_sh, &ctl_word(w.counts, kWaveFetch + ((parts & 1u) ? 0 : 1)), launch_stack(smem_stack, scap, spill, total),
      steps, st, st_sh, lerr);
  if (kStats) {
    warp_count(&ctr->nodes, st.nodes);
    warp_count(&ctr->leaves, st.leaves);
    warp_count(&ctr->tris, st.tris);
    warp_count(&ctr->ext_rays, st.rays);
    warp_count(&ctr->shadow_nodes, st_sh.nodes);
    warp_count(&ctr->shadow_leaves, st_sh.leaves);
    warp_count(&ctr->shadow_tris, st_sh.tris);
    warp_count(&ctr->shadow_rays, st_sh.rays);
  }
  if (lerr) atomicOr(err, lerr);
}

// ======================================================================= SDF
// One sphere-tracing step per lane and call, lanes refilled as their queries
// finish, so a warp is not held by its longest march (inside the shading stage
// the marches took nine tenths of a frame of the SDF gallery).

__device__ __forceinline__ void flush_sdf(DevCounters* ctr, const SdfCount& c) {
  warp_count(&ctr->sdf_tests, c.tests);
  warp_count(&ctr->sdf_steps, c.steps);
  warp_count(&ctr->sdf_hits, c.hits);
}

__global__ void __launch_bounds__(256) k_sdf(DevScene s, WaveState w, const uint32_t* q, uint32_t depth,
                                             DevCounters* ctr) {
  const uint32_t n = ctl_word(w.counts, kWaveExt + (depth & 1u));
  SdfCount c;
  const WaveSdfExtSource src{s.sdf, s.sdf_count, q, w.ray_o, w.ray_d, w.hit};
  sdf_persistent<WaveSdfExtSource, false>(src, n, &ctl_word(w.counts, kWaveFetchSdf), kSdfSteps, c);
  flush_sdf(ctr, c);
}

__global__ void __launch_bounds__(256) k_sdf_shadow(DevScene s, WaveState w, uint32_t depth, DevCounters* ctr) {
  const uint32_t n = ctl_word(w.counts, kWaveShadow + (depth & 1u));
  SdfCount c;
  const WaveSdfShadowSource src{s.sdf, s.sdf_count, w.sh_o, w.sh_d, w.sh_path};
  sdf_persistent<WaveSdfShadowSource, true>(src, n, &ctl_word(w.counts, kWaveFetchSdfShadow), kSdfSteps, c);
  flush_sdf(ctr, c);
}

// ===================================================================== shade
// Variants as in the loop driver: code no path of the scene can reach
// (procedural effects, SDF hits, transmissive / clear-coat / sheen / toon
// materials and the environment map) is compiled out, because the stage waits
// on instruction fetch and on chains of loads.  64 registers: at 80 (24 warps per
// SM instead of 32, spills 28 to 64 bytes fewer) a full-HD frame of the grid took
// 19.7 ms instead of 18.3, at 48 19.0.
template <bool kParity, bool kEffects, bool kSdf, bool kExotic>
__global__ void __launch_bounds__(256, 4) k_shade(DevScene s, DevSettings st, WaveState w, const uint32_t* q,
                                                  uint32_t* qn, uint32_t depth, DevCounters* ctr) {
  const uint32_t cur = depth & 1u;
  const uint32_t n = ctl_word(w.counts, kWaveExt + cur);
  if (blockIdx.x == 0 && threadIdx.x == 0) {   // the next trace stage claims from 0
    ctl_word(w.counts, kWaveFetch) = 0u;
    ctl_word(w.counts, kWaveFetch + 1) = 0u;
  }
  uint32_t shadow_tests = 0u;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const uint32_t j = base + threadIdx.x;
    uint32_t p = 0u;
    ShadeOut R;
    R.next = R.shadow = false;
    if (j < n) {
      p = q[j];
      const float4 o4 = w.ray_o[p], d4 = w.ray_d[p], t4 = w.thr[p], r4 = w.rad[p];
      const float2 h2 = w.hit[p];
      PathRegs P;
      P.o = mk(o4.x, o4.y, o4.z);
      P.d = mk(d4.x, d4.y, d4.z);
      P.thr = mk(t4.x, t4.y, t4.z);
      P.rad = mk(r4.x, r4.y, r4.z);
      P.segs = r4.w;
      P.rng = w.rng[p];
      R = shade_bounce<kParity, kEffects, kSdf, kExotic, true>(s, st, s.lights, depth, P, h2.x, __float_as_uint(h2.y));
      if (R.next) {
        w.ray_o[p] = make_float4(P.o.x, P.o.y, P.o.z, 0.0f);
        w.ray_d[p] = make_float4(P.d.x, P.d.y, P.d.z, 0.0f);
        w.thr[p] = make_float4(P.thr.x, P.thr.y, P.thr.z, 0.0f);
        w.rng[p] = P.rng;
      }
      w.rad[p] = make_float4(P.rad.x, P.rad.y, P.rad.z, P.segs);
      shadow_tests += R.shadow_tests;
    }
    // Warp-aggregated appends (the whole warp reaches these together).
    const uint32_t slot_n = warp_append(&ctl_word(w.counts, kWaveExt + (cur ^ 1u)), R.next);
    if (R.next) qn[slot_n] = p;
    const uint32_t slot_s = warp_append(&ctl_word(w.counts, kWaveShadow + cur), R.shadow);
    if (R.shadow) {
      w.sh_path[slot_s] = p;
      w.sh_o[slot_s] = make_float4(R.sh_o.x, R.sh_o.y, R.sh_o.z, R.sh_t);
      w.sh_d[slot_s] = make_float4(R.sh_d.x, R.sh_d.y, R.sh_d.z, 0.0f);
      w.sh_c[slot_s] = make_float4(R.sh_c.x, R.sh_c.y, R.sh_c.z, 0.0f);
    }
  }
  warp_count(&ctr->shadow_tests, shadow_tests);
}

// Scenes with transmissive materials and SDF primitives: each shadow query's
// closest-hit loop tests the SDF primitives after the triangles (one query per
// thread; scenes without SDF primitives take these queries in k_trace).
template <bool kStats, bool kWt>
__global__ void __launch_bounds__(256) k_shadow_transmissive(DevScene s, WaveState w, uint32_t depth, int cap,
                                                             DevCounters* ctr, uint32_t* err) {
  extern __shared__ int2 smem_stack[];
  const TwoLevelStack stk = smem_stack_of(smem_stack + threadIdx.x, static_cast<int>(blockDim.x), cap);
  const uint32_t n = ctl_word(w.counts, kWaveShadow + (depth & 1u));
  uint32_t local_err = 0u;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const uint32_t j = base + threadIdx.x;
    TraceStats st;
    SdfCount sdf_n;
    if (j < n) {
      const float4 o4 = w.sh_o[j], d4 = w.sh_d[j];
      V3 so = mk(o4.x, o4.y, o4.z);
      const V3 sd = mk(d4.x, d4.y, d4.z);
      float remain = o4.w;
      bool visible = true;
      // Closest-hit loop that steps through up to 8 transmissive occluders
      // (src/pathtracer/ScalarCpuPathTracer.cpp:1067-1087).
      for (uint32_t skips = 0; skips < 8u && remain > 0.004f; ++skips) {
        float t;
        uint32_t prim;
        trace_closest<kStats, kWt>(s, so, sd, stk, t, prim, st, local_err);
        if (s.sdf_count != 0u) sdf_closest(s.sdf, s.sdf_count, so, sd, t, prim, sdf_n);
        if (prim == kMiss || t >= remain) break;
        const uint32_t mat_index = (prim & kSdfTag) ? sdf_material(s.sdf, prim & ~kSdfTag)
                                                    : __float_as_uint(__ldg(s.shade + prim).w);
        const uint32_t mi = mat_index < s.material_count - 1u ? mat_index : s.material_count - 1u;
        const float* mm = s.materials + 16u * mi;
        const bool tr = static_cast<uint32_t>(mm[7] + 0.5f) == 5u || mm[10] > 0.05f;
        if (!tr) {
          visible = false;
          break;
        }
        const float adv = t + 0.004f;
        so = add(so, mul(sd, adv));
        remain -= adv;
      }
      if (visible) {
        const uint32_t p = w.sh_path[j];
        const float4 c = w.sh_c[j];
        float4 r = w.rad[p];
        r.x = r.x + c.x;
        r.y = r.y + c.y;
        r.z = r.z + c.z;
        w.rad[p] = r;
      }
    }
    if (kStats) {
      warp_count(&ctr->shadow_nodes, st.nodes);
      warp_count(&ctr->shadow_leaves, st.leaves);
      warp_count(&ctr->shadow_tris, st.tris);
      warp_count(&ctr->shadow_rays, j < n ? 1u : 0u);
    }
    if (s.sdf_count != 0u) {
      warp_count(&ctr->sdf_tests, sdf_n.tests);
      warp_count(&ctr->sdf_steps, sdf_n.steps);
      warp_count(&ctr->sdf_hits, sdf_n.hits);
    }
  }
  if (local_err) atomicOr(err, local_err);
}

// ================================================================ accumulate
__global__ void __launch_bounds__(256) k_accumulate(DevSettings st, WaveState w, WaveTile tile, Film film,
                                                    DevCounters* ctr) {
  const uint32_t tile_px = tile.w * tile.h;
  uint32_t samples = 0u, segs = 0u, dropped = 0u;
  for (uint32_t base = blockIdx.x * blockDim.x; base < tile_px; base += gridDim.x * blockDim.x) {
    const uint32_t k = base + threadIdx.x;
    if (k < tile_px) {
      const uint32_t pl = tile_order_pixel(k, tile.w, tile.h);
      const uint32_t x = tile.x + pl % tile.w, y = tile.y + pl / tile.w;
      const size_t px = static_cast<size_t>(y) * film.width + x;
      float4 acc = film.sum[px];
      uint32_t cnt = film.count[px];
      for (uint32_t sl = 0; sl < tile.sample_count; ++sl) {
        const float4 r = w.rad[wave_slot(k, sl, tile_px, tile.sample_count)];
        if (!(isfinite(r.x) && isfinite(r.y) && isfinite(r.z))) {
          ++dropped;   // dropped before the film, like the reference's shade_pixel
          continue;
        }
        float cx = r.x, cy = r.y, cz = r.z;
        if (st.firefly_clamp > 0.0f) {
          cx = smin(cx, st.firefly_clamp);
          cy = smin(cy, st.firefly_clamp);
          cz = smin(cz, st.firefly_clamp);
        }
        acc.x = acc.x + cx;
        acc.y = acc.y + cy;
        acc.z = acc.z + cz;
        ++cnt;
        ++samples;
        segs += static_cast<uint32_t>(r.w);
      }
      film.sum[px] = acc;
      film.count[px] = cnt;
    }
  }
  block_count3(&ctr->samples, samples, &ctr->rays, segs, &ctr->dropped, dropped);
}

namespace {

using TraceFn = void (*)(DevScene, WaveState, const uint32_t*, uint32_t, uint32_t, int, int2*, int, int, DevCounters*,
                         uint32_t*);
// [stats][watertight][transmissive shadow queries]
TraceFn trace_fn(bool stats, bool wt, bool trans) {
  static const TraceFn t[2][2][2] = {
      {{k_trace<false, false, false>, k_trace<false, false, true>}, {k_trace<false, true, false>, k_trace<false, true, true>}},
      {{k_trace<true, false, false>, k_trace<true, false, true>}, {k_trace<true, true, false>, k_trace<true, true, true>}}};
  return t[stats ? 1 : 0][wt ? 1 : 0][trans ? 1 : 0];
}

using ShadeFn = void (*)(DevScene, DevSettings, WaveState, const uint32_t*, uint32_t*, uint32_t, DevCounters*);
template <bool kP, bool kE>
ShadeFn shade_fn_pe(bool sdf, bool exotic) {
  static const ShadeFn t[2][2] = {{k_shade<kP, kE, false, false>, k_shade<kP, kE, false, true>},
                                  {k_shade<kP, kE, true, false>, k_shade<kP, kE, true, true>}};
  return t[sdf ? 1 : 0][exotic ? 1 : 0];
}
ShadeFn shade_fn(bool parity, bool effects, bool sdf, bool exotic) {
  if (parity) return effects ? shade_fn_pe<true, true>(sdf, exotic) : shade_fn_pe<true, false>(sdf, exotic);
  return effects ? shade_fn_pe<false, true>(sdf, exotic) : shade_fn_pe<false, false>(sdf, exotic);
}

}  // namespace

// Per wave: raygen, then per depth one trace and one shade launch (the shadow
// queries of a depth are traced with the next depth's extension rays; the last
// depth queues none), then the film.  The launches a scene with SDF primitives
// adds: its closest hits after the trace, its occlusion of the shadow queries
// after the shading -- or, with transmissive materials, their whole loop there.
cudaError_t LaunchWave(const DevScene& s, const DevSettings& st, const WaveState& w, const WaveTile& tile,
                       const Film& film, bool parity, bool stats, const LaunchShape& ls, DevCounters* ctr,
                       uint32_t* err, StageTimer* timer) {
  const size_t smem = StackSmemBytes(ls.block, ls.smem_entries);
  const size_t smem_full = StackSmemBytes(ls.block, ls.stack_cap);
  const bool sdf = s.sdf_count != 0u, wt = s.watertight != 0u;
  const bool trans_sdf = sdf && s.has_transmissive;   // shadow queries by k_shadow_transmissive
  const TraceFn trace = trace_fn(stats, wt, s.has_transmissive && !sdf);
  const ShadeFn shade = shade_fn(parity, s.has_effects, sdf, s.has_exotic || s.env_map != nullptr);
  StageTimer dummy;
  StageTimer& tm = timer ? *timer : dummy;
  tm.begin(0, ls.stream);
  if (parity) k_raygen<true><<<ls.grid, ls.block, 0, ls.stream>>>(s, st, w, tile);
  else k_raygen<false><<<ls.grid, ls.block, 0, ls.stream>>>(s, st, w, tile);
  tm.end(ls.stream);
  for (uint32_t depth = 0; depth < st.max_depth; ++depth) {
    const uint32_t* q = w.q[depth & 1u];
    const bool queries = depth > 0u && st.enable_nee && !trans_sdf;   // the previous depth's shadow queries
    auto run_trace = [&](uint32_t parts) {
      trace<<<ls.grid, ls.block, smem, ls.stream>>>(s, w, q, depth, parts, ls.smem_entries, ls.spill, ls.stack_cap,
                                                    ls.steps, ctr, err);
    };
    if (timer && queries) {   // stage timing separates the two kinds of query
      tm.begin(3, ls.stream);
      run_trace(2u);
      tm.end(ls.stream);
    }
    tm.begin(1, ls.stream);
    run_trace(queries && !timer ? 3u : 1u);
    if (sdf) k_sdf<<<ls.grid, ls.block, 0, ls.stream>>>(s, w, q, depth, ctr);
    tm.end(ls.stream);
    tm.begin(2, ls.stream);
    shade<<<ls.grid, ls.block, 0, ls.stream>>>(s, st, w, q, w.q[(depth & 1u) ^ 1u], depth, ctr);
    tm.end(ls.stream);
    if (st.enable_nee && sdf) {
      tm.begin(3, ls.stream);
      if (!trans_sdf) k_sdf_shadow<<<ls.grid, ls.block, 0, ls.stream>>>(s, w, depth, ctr);
#define VKPTC_SHT(S, W) \
  k_shadow_transmissive<S, W><<<ls.grid, ls.block, smem_full, ls.stream>>>(s, w, depth, ls.stack_cap, ctr, err)
      else if (wt && stats) VKPTC_SHT(true, true);
      else if (wt) VKPTC_SHT(false, true);
      else if (stats) VKPTC_SHT(true, false);
      else VKPTC_SHT(false, false);
#undef VKPTC_SHT
      tm.end(ls.stream);
    }
  }
  tm.begin(4, ls.stream);
  k_accumulate<<<ls.grid, ls.block, 0, ls.stream>>>(st, w, tile, film, ctr);
  tm.end(ls.stream);
  return cudaGetLastError();
}

// ==================================================================== film
__global__ void k_resolve_hdr(Film film, float* out) {
  const size_t npx = static_cast<size_t>(film.width) * film.height;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < npx;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t c = film.count[i];
    const float inv = 1.0f / static_cast<float>(c > 1u ? c : 1u);
    const float4 v = film.sum[i];
    out[3 * i + 0] = v.x * inv;
    out[3 * i + 1] = v.y * inv;
    out[3 * i + 2] = v.z * inv;
  }
}

__global__ void k_pack_film(const float4* __restrict__ sum, size_t npx, float* __restrict__ out) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < npx;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const float4 v = sum[i];
    out[3 * i + 0] = v.x;
    out[3 * i + 1] = v.y;
    out[3 * i + 2] = v.z;
  }
}

__global__ void __launch_bounds__(256) k_read_probe(const float4* __restrict__ buf, size_t n, uint32_t reps,
                                                     float* sink) {
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  float acc = 0.0f;
  for (uint32_t r = 0; r < reps; ++r) {
    size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    for (; i + 3 * stride < n; i += 4 * stride) {
      const float4 a = __ldcg(buf + i), b = __ldcg(buf + i + stride);
      const float4 c = __ldcg(buf + i + 2 * stride), d = __ldcg(buf + i + 3 * stride);
      acc += (a.x + b.y) + (c.z + d.w);
    }
    for (; i < n; i += stride) acc += __ldcg(buf + i).x;
  }
  if (acc == -1.0e30f) sink[0] = acc;   // keeps the loads; the buffer holds zeros
}

cudaError_t LaunchReadProbe(const float4* buf, size_t bytes, uint32_t reps, int grid, float* sink,
                            cudaStream_t stream) {
  k_read_probe<<<grid, 256, 0, stream>>>(buf, bytes / 16u, reps, sink);
  return cudaGetLastError();
}

cudaError_t LaunchPackFilm(const Film& film, float* rgb_out, cudaStream_t stream) {
  const size_t npx = static_cast<size_t>(film.width) * film.height;
  const int grid = static_cast<int>(std::min<size_t>(8192, std::max<size_t>(1, (npx + 255) / 256)));
  k_pack_film<<<grid, 256, 0, stream>>>(film.sum, npx, rgb_out);
  return cudaGetLastError();
}

// One block per instance range (strided), its threads over the range.
__global__ void k_set_instance_materials(float4* __restrict__ shade, const uint4* __restrict__ ranges,
                                         uint32_t range_count) {
  for (uint32_t r = blockIdx.x; r < range_count; r += gridDim.x) {
    const uint4 g = ranges[r];
    const float m = __uint_as_float(g.z);
    for (uint32_t k = threadIdx.x; k < g.y; k += blockDim.x) shade[g.x + k].w = m;
  }
}

cudaError_t LaunchSetInstanceMaterials(float4* shade, const uint4* ranges, uint32_t range_count, cudaStream_t stream) {
  if (range_count == 0u) return cudaSuccess;
  const int grid = static_cast<int>(std::min<uint32_t>(range_count, 148u * 8u));
  k_set_instance_materials<<<grid, 256, 0, stream>>>(shade, ranges, range_count);
  return cudaGetLastError();
}

// ApplyFilmResolve (src/pathtracer/FilmBuffer.cpp:253-325) per pixel, on the
// film's per-pixel mean: exposure then white balance, non-finite to 0, tone
// map, gamma (pow, FP64 rounded once in parity mode), clamp, and the x86
// float -> uint8 conversion (truncate to int32, keep the low byte).
__device__ __forceinline__ float ldr_tonemap(float x, uint32_t mode) {
  switch (mode) {
    case 1u:
      return x / (1.0f + x);
    case 2u: {
      const float A = 0.15f, B = 0.50f, C = 0.10f, D = 0.20f, E = 0.02f, F = 0.30f;
      const float W = 11.2f;
      const float fx = ((x * (A * x + C * B) + D * E) / (x * (A * x + B) + D * F)) - E / F;
      const float fw = ((W * (A * W + C * B) + D * E) / (W * (A * W + B) + D * F)) - E / F;
      return fx / fw;
    }
    case 3u:
      return (x * (2.51f * x + 0.03f)) / (x * (2.43f * x + 0.59f) + 0.14f);
    default:
      return x;
  }
}

template <bool kParity>
__global__ void k_resolve_ldr(Film film, LdrResolve rs, uint8_t* __restrict__ out) {
  const size_t npx = static_cast<size_t>(film.width) * film.height;
  const float inv_gamma = 1.0f / smax(0.01f, rs.gamma);
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < npx;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t c = film.count[i];
    const float inv = 1.0f / static_cast<float>(c > 1u ? c : 1u);
    const float4 v = film.sum[i];
    float ch[3] = {v.x * inv * rs.exposure * rs.wb[0], v.y * inv * rs.exposure * rs.wb[1],
                   v.z * inv * rs.exposure * rs.wb[2]};
    uint32_t word = 0xFF000000u;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float x = ch[k];
      if (!isfinite(x)) x = 0.0f;
      x = ldr_tonemap(x, rs.tone_map);
      if (rs.output_transform == 0u) {
        const float b = smax(0.0f, x);
        x = kParity ? parity_pow(b, inv_gamma) : powf(b, inv_gamma);
      }
      if (rs.clamp_output) x = smin(1.0f, smax(0.0f, x));
      const int32_t q = __float2int_rz(x * 255.0f + 0.5f);
      word |= (static_cast<uint32_t>(q) & 0xFFu) << (8 * k);
    }
    reinterpret_cast<uint32_t*>(out)[i] = word;
  }
}

cudaError_t LaunchResolveLdr(const Film& film, const LdrResolve& rs, bool parity, uint8_t* rgba_out,
                             cudaStream_t stream) {
  const size_t npx = static_cast<size_t>(film.width) * film.height;
  const int grid = static_cast<int>(std::min<size_t>(4096, std::max<size_t>(1, (npx + 255) / 256)));
  if (parity) k_resolve_ldr<true><<<grid, 256, 0, stream>>>(film, rs, rgba_out);
  else k_resolve_ldr<false><<<grid, 256, 0, stream>>>(film, rs, rgba_out);
  return cudaGetLastError();
}

cudaError_t ConfigureStackSmem() {
  cudaError_t e = cudaSuccess;
  const auto all = [&](auto wt) {
    constexpr bool W = decltype(wt)::value;
    if (e == cudaSuccess) e = allow_full_smem(k_trace_rays<true, true, W>);
    if (e == cudaSuccess) e = allow_full_smem(k_trace_rays<true, false, W>);
    if (e == cudaSuccess) e = allow_full_smem(k_trace_rays<false, true, W>);
    if (e == cudaSuccess) e = allow_full_smem(k_trace_rays<false, false, W>);
    if (e == cudaSuccess) e = allow_full_smem(k_trace<true, W, false>);
    if (e == cudaSuccess) e = allow_full_smem(k_trace<true, W, true>);
    if (e == cudaSuccess) e = allow_full_smem(k_trace<false, W, false>);
    if (e == cudaSuccess) e = allow_full_smem(k_trace<false, W, true>);
    if (e == cudaSuccess) e = allow_full_smem(k_shadow_transmissive<true, W>);
    if (e == cudaSuccess) e = allow_full_smem(k_shadow_transmissive<false, W>);
  };
  all(std::false_type{});
  all(std::true_type{});
  return e;
}

int ExtendBlocksPerSm(int block, size_t smem, bool watertight) {
  int blocks = 0;
  const cudaError_t e = watertight
      ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_trace<false, true, false>, block, smem)
      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_trace<false, false, false>, block, smem);
  if (e != cudaSuccess) return 1;
  return blocks > 0 ? blocks : 1;
}

cudaError_t LaunchResolveHdr(const Film& film, float* rgb_out, cudaStream_t stream) {
  k_resolve_hdr<<<592, 256, 0, stream>>>(film, rgb_out);
  return cudaGetLastError();
}

}  // namespace vkptc
