// adjoint.cu -- forward / loss / backward kernels of differentiable rendering.
//
// Forward: the renderer's trace and next-event arithmetic (adjoint.cuh) in the
// reference's operation order, so each sample's radiance equals the renderer's
// (the film test pins this bit-for-bit).  Up to one path per resident thread
// it is one thread per (sample, pixel) path with inline traversal; above, a
// wavefront that writes the vertex records (AdjTraceSource below).
//
// Backward: from those records, or, where the forward did not write them,
// "re-trace from the seed": the same path is replayed from its RNG key,
// recording per vertex the ray, hit, throughput, roulette divisor, RNG state
// and decision flags (64 bytes, at most 8 vertices).  The records are swept in
// reverse with each vertex's vector-Jacobian product (adj_vertex_vjp); albedo
// and emission enter affinely.  Per-vertex parameter gradients are added in a
// fixed order to per-warp shared-memory slots, then per-block partials, then a
// fixed-order FP64 reduction: the gradient is deterministic for a given launch
// shape.
#define VKPTC_INLINE_UNIT 1   // common.cuh
#include "adjoint.cuh"
#include <algorithm>

#include "adjoint_launch.h"
#include "traverse.cuh"

namespace vkptc {

namespace {

struct AdjRec {
  float4 a;   // origin xyz, hit distance
  float4 b;   // direction xyz, primitive bits (kMiss on a miss)
  float4 c;   // throughput at the vertex xyz, roulette divisor applied after it
  uint4 e;    // RNG state lo, hi at the vertex, flags, material index
};
static_assert(sizeof(AdjRec) == kAdjRecordFloat4s * sizeof(float4), "record layout of the backward buffers");
static_assert(kAdjVertexSlots == kAdjMaxDepth, "record slots per path");

__device__ __forceinline__ uint32_t mat_slot(const DevScene& s, uint32_t mat_index) {
  return mat_index < s.material_count - 1u ? mat_index : s.material_count - 1u;
}

// The primal path of pixel (x, y), sample `sample`.  kRecord keeps the
// vertex records for the reverse sweep: vertex k at rec[k * rec_stride].  Returns radiance xyz and, in w, the
// bits of a 32-bit hash of the path's discrete decisions (hit primitives and
// vertex flags): two evaluations with equal hashes took the same branches.
template <bool kParity, bool kRecord>
__device__ __forceinline__ float4 adj_primal(const DevScene& s, const DevSettings& st, const float* mat0,
                                             uint32_t x, uint32_t y, uint32_t sample, const TwoLevelStack& stk,
                                             uint32_t& err, AdjRec* rec, uint32_t& nrec, uint32_t rec_stride = 1u) {
  V3 o, d;
  uint64_t rng;
  camera_path<kParity>(s, st, x, y, sample, o, d, rng);
  V3 thr = mk(1.0f, 1.0f, 1.0f), thr0 = thr, rad = mk(0.0f, 0.0f, 0.0f);
  uint64_t sig = 0u;
  nrec = 0u;
  const float* lights = s.lights;
  TraceStats ts;
  for (uint32_t depth = 0; depth < st.max_depth; ++depth) {
    float t;
    uint32_t prim;
    trace_closest<false>(s, o, d, stk, t, prim, ts, err);
    if (prim == kMiss) {
      rad = add(rad, mulv(thr, s.env));
      sig = mix64(sig ^ 0xFFFFFFFFull);
      if (kRecord) {
        AdjRec& r = rec[static_cast<size_t>(nrec++) * rec_stride];
        r.a = make_float4(o.x, o.y, o.z, 0.0f);
        r.b = make_float4(d.x, d.y, d.z, __uint_as_float(kMiss));
        r.c = make_float4(thr.x, thr.y, thr.z, 1.0f);
        r.e = make_uint4(0u, 0u, kVfMiss, 0u);
      }
      break;
    }
    const uint64_t rng_at = rng;
    const V3 o_at = o, d_at = d;
    const float4 sh = __ldg(s.shade + prim);
    const V3 gn = mk(sh.x, sh.y, sh.z);
    const uint32_t mi = mat_slot(s, __float_as_uint(sh.w));
    const MaterialRec m = load_material(s.materials + 16u * mi);
    uint32_t flags = 0u;
    AdjVertex R;
    adj_vertex<kParity>(s, st, lights, depth, o, d, t, gn, m, clamp01(m.roughness), rng, flags, R);
    // emission, then the next-event term, in the renderer's order
    const bool emissive_model = m.model == 1u || m.emissive.x > 0.0f || m.emissive.y > 0.0f || m.emissive.z > 0.0f;
    if (!st.enable_nee || depth == 0u) rad = add(rad, mulv(thr, m.emissive));
    else if (st.enable_mis && emissive_model) rad = add(rad, mul(mulv(thr, m.emissive), R.w_e));
    if (R.nee) {
      const V3 c = st.enable_mis ? mul(mulv(thr, R.q.radiance), R.w_n) : mulv(thr, R.q.radiance);
      bool vis = true;
      if (R.q.remain > 0.004f) vis = !trace_any<false>(s, R.q.origin, R.q.dir, R.q.remain, stk, ts, err);
      if (vis) {
        rad = add(rad, c);
        flags |= kVfNeeVis;
      }
    }
    const V3 thr_at = thr;
    float rr = 1.0f;
    bool cont = false;
    if (R.scattered) {
      const V3 wgt = albedo_effect0(m);
      const V3 wgt0 = albedo_effect0(load_material(mat0 + 16u * mi));
      thr = mulv(thr, wgt);
      thr0 = mulv(thr0, wgt0);
      const float tmx = smax(thr0.x, smax(thr0.y, thr0.z));
      if (!(tmx < 0.001f)) {
        rr = smin(st.rr_max, smax(st.rr_min, tmx));
        if (!(depth >= st.rr_start && next01(rng) > rr)) {
          thr = divs(thr, rr);
          thr0 = divs(thr0, rr);
          cont = depth + 1u < st.max_depth;
          o = add(R.hp, mul(R.out, 0.002f));
          d = R.out;
        }
      }
    }
    sig = mix64(sig ^ (static_cast<uint64_t>(prim + 1u) | (static_cast<uint64_t>(flags | (cont ? kVfCont : 0u)) << 32)));
    if (kRecord) {
      AdjRec& r = rec[static_cast<size_t>(nrec++) * rec_stride];
      r.a = make_float4(o_at.x, o_at.y, o_at.z, t);
      r.b = make_float4(d_at.x, d_at.y, d_at.z, __uint_as_float(prim));
      r.c = make_float4(thr_at.x, thr_at.y, thr_at.z, rr);
      r.e = make_uint4(static_cast<uint32_t>(rng_at), static_cast<uint32_t>(rng_at >> 32),
                       flags | (cont ? kVfCont : 0u), mi);
    }
    if (!cont) break;
  }
  return make_float4(rad.x, rad.y, rad.z, __uint_as_float(static_cast<uint32_t>(sig ^ (sig >> 32))));
}

// One path per thread from start to end: the forward without records, and the
// recording forward of few paths.  102 registers (5 blocks of 128 threads per
// SM): 1.98 -> 1.87 ms per 524,288-path forward.  kRecord: every path's vertex
// records (recs, the backward's layout with all paths as one chunk) and their
// count (nrec), so a backward over the same paths needs no replay.
template <bool kParity, bool kRecord>
__global__ void __launch_bounds__(128, 5) k_adj_forward(DevScene s, DevSettings st, const float* mat0, uint32_t spp,
                                                     uint32_t first_sample, int cap, float4* rad, AdjRec* recs,
                                                     uint32_t* nrec_out, uint32_t* err) {
  extern __shared__ int2 smem_stack[];
  const TwoLevelStack stk = smem_stack_of(smem_stack + threadIdx.x, static_cast<int>(blockDim.x), cap);
  const uint32_t npx = st.width * st.height;
  const uint64_t n = static_cast<uint64_t>(npx) * spp;
  uint32_t local_err = 0u;
  for (uint64_t j = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; j < n;
       j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t sl = static_cast<uint32_t>(j / npx), p = static_cast<uint32_t>(j % npx);
    uint32_t nrec = 0u;
    if (kRecord) {
      rad[j] = adj_primal<kParity, true>(s, st, mat0, p % st.width, p / st.width, first_sample + sl, stk, local_err,
                                         recs + j, nrec, static_cast<uint32_t>(n));
      nrec_out[j] = nrec;
    } else {
      rad[j] = adj_primal<kParity, false>(s, st, mat0, p % st.width, p / st.width, first_sample + sl, stk, local_err,
                                          nullptr, nrec);
    }
  }
  if (local_err) atomicOr(err, local_err);
}

// ------------------------------------------------------------ recording forward
// The recording forward of many paths runs as a wavefront, as the renderer's frames do
// (kernels.cu): per depth one trace launch (the closest hits of this depth's
// paths and the previous depth's next-event queries) and one shading launch,
// which writes the vertex records.  Walking a whole path per thread leaves a warp
// waiting for its longest path, with the traversal and the shading code in one
// kernel at 96 registers: 1.38 ms per 524,288-path forward, this takes 0.84 ms.
// Words of AdjWave::counts: 0, 1 extension queue sizes, 2, 3 query counts by the
// depth that fills them (even, odd), 4 the trace's fetch counter.
struct AdjTraceSource {
  GeoView geo;
  const uint32_t* q;
  AdjWave w;
  float4* rad;
  AdjRec* rec_prev;     // the previous depth's vertex of every path
  uint32_t n_ext;
  static constexpr bool kUniform = true;
  __device__ __forceinline__ const GeoView& geo_at(uint32_t) const { return geo; }
  __device__ __forceinline__ bool any(uint32_t j) const { return j >= n_ext; }
  __device__ __forceinline__ void load(uint32_t j, V3& o, V3& d, float& tm, GeoView& g) const {
    g = geo;
    const bool sh = j >= n_ext;
    const uint32_t k = sh ? j - n_ext : q[j];
    const float4 a = (sh ? w.sh_o : w.ray_o)[k], b = (sh ? w.sh_d : w.ray_d)[k];
    o = mk(a.x, a.y, a.z);
    d = mk(b.x, b.y, b.z);
    tm = sh ? a.w : kInf;
  }
  __device__ __forceinline__ bool finish(uint32_t j, float t, uint32_t prim, V3&, V3, float&) const {
    if (j < n_ext) {
      w.hit[q[j]] = make_float2(t, __uint_as_float(prim));
      return false;
    }
    if (prim) return false;   // occluded
    const uint32_t p = w.sh_path[j - n_ext];
    const float4 c = w.sh_c[j - n_ext];
    float4 r = rad[p];
    r.x = r.x + c.x;
    r.y = r.y + c.y;
    r.z = r.z + c.z;
    rad[p] = r;
    rec_prev[p].e.z |= kVfNeeVis;
    return false;
  }
};

template <bool kParity>
__global__ void __launch_bounds__(256) k_adj_raygen(DevScene s, DevSettings st, uint32_t n, uint32_t first_sample,
                                                    AdjWave w, float4* rad) {
  const uint32_t npx = st.width * st.height;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const uint32_t sl = j / npx, p = j - sl * npx;
    V3 o, d;
    uint64_t rng;
    camera_path<kParity>(s, st, p % st.width, p / st.width, first_sample + sl, o, d, rng);
    w.rng[j] = rng;
    w.ray_o[j] = make_float4(o.x, o.y, o.z, 0.0f);
    w.ray_d[j] = make_float4(d.x, d.y, d.z, 0.0f);
    w.thr[j] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    w.thr0[j] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    rad[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    w.q[0][j] = j;
  }
  if (blockIdx.x == 0 && threadIdx.x < 8u) ctl_word(w.counts, threadIdx.x) = threadIdx.x == 0u ? n : 0u;
}

__global__ void __launch_bounds__(256, 4) k_adj_trace(DevScene s, AdjWave w, const uint32_t* q, uint32_t depth,
                                                      float4* rad, AdjRec* rec_prev, int scap, int2* spill, int total,
                                                      int steps, uint32_t* err) {
  extern __shared__ int2 smem_stack[];
  const uint32_t cur = depth & 1u;
  const uint32_t n_ext = ctl_word(w.counts, cur), n_sh = depth > 0u ? ctl_word(w.counts, 2u + (cur ^ 1u)) : 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl_word(w.counts, cur ^ 1u) = 0u;
    ctl_word(w.counts, 2u + cur) = 0u;
  }
  const AdjTraceSource src{geo_of(s), q, w, rad, rec_prev, n_ext};
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const TwoLevelStack stk{smem_stack + threadIdx.x, static_cast<int>(blockDim.x), scap, spill ? spill + gtid : nullptr,
                          static_cast<int>(gridDim.x * blockDim.x), total};
  TraceStats st;
  uint32_t lerr = 0u;
  persistent_traverse<AdjTraceSource, kQueryMixed, false>(src, n_ext + n_sh, &ctl_word(w.counts, 4), stk, steps, st, st, lerr);
  if (lerr) atomicOr(err, lerr);
}

// One vertex per queued path: adj_primal's bounce with the visibility test left
// to the next trace, the record written, survivors and queries appended.
template <bool kParity>
__global__ void __launch_bounds__(128, 5) k_adj_shade(DevScene s, DevSettings st, const float* mat0, AdjWave w,
                                                      const uint32_t* q, uint32_t* qn, uint32_t depth, float4* rad,
                                                      AdjRec* rec, uint32_t* nrec) {
  const uint32_t cur = depth & 1u;
  const uint32_t n = ctl_word(w.counts, cur);
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl_word(w.counts, 4) = 0u;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const uint32_t j = base + threadIdx.x;
    bool next = false, shadow = false;
    uint32_t p = 0u;
    V3 sh_c = mk(0.0f, 0.0f, 0.0f);
    AdjVertex R;
    R.nee = false;
    if (j < n) {
      p = q[j];
      const float4 o4 = w.ray_o[p], d4 = w.ray_d[p], t4 = w.thr[p], u4 = w.thr0[p], r4 = rad[p];
      const float2 h2 = w.hit[p];
      const V3 o = mk(o4.x, o4.y, o4.z), d = mk(d4.x, d4.y, d4.z);
      V3 thr = mk(t4.x, t4.y, t4.z), thr0 = mk(u4.x, u4.y, u4.z), r = mk(r4.x, r4.y, r4.z);
      const uint32_t prim = __float_as_uint(h2.y);
      AdjRec v;
      v.a = make_float4(o.x, o.y, o.z, prim == kMiss ? 0.0f : h2.x);
      v.b = make_float4(d.x, d.y, d.z, h2.y);
      if (prim == kMiss) {
        r = add(r, mulv(thr, s.env));
        v.c = make_float4(thr.x, thr.y, thr.z, 1.0f);
        v.e = make_uint4(0u, 0u, kVfMiss, 0u);
      } else {
        uint64_t rng = w.rng[p];
        const uint64_t rng_at = rng;
        const float4 sh = __ldg(s.shade + prim);
        const V3 gn = mk(sh.x, sh.y, sh.z);
        const uint32_t mi = mat_slot(s, __float_as_uint(sh.w));
        const MaterialRec m = load_material(s.materials + 16u * mi);
        uint32_t flags = 0u;
        adj_vertex<kParity>(s, st, s.lights, depth, o, d, h2.x, gn, m, clamp01(m.roughness), rng, flags, R);
        const bool emissive_model = m.model == 1u || m.emissive.x > 0.0f || m.emissive.y > 0.0f || m.emissive.z > 0.0f;
        if (!st.enable_nee || depth == 0u) r = add(r, mulv(thr, m.emissive));
        else if (st.enable_mis && emissive_model) r = add(r, mul(mulv(thr, m.emissive), R.w_e));
        if (R.nee) {
          sh_c = st.enable_mis ? mul(mulv(thr, R.q.radiance), R.w_n) : mulv(thr, R.q.radiance);
          shadow = R.q.remain > 0.004f;
          if (!shadow) {   // no visibility test runs for so short a segment
            r = add(r, sh_c);
            flags |= kVfNeeVis;
          }
        }
        v.c = make_float4(thr.x, thr.y, thr.z, 1.0f);
        if (R.scattered) {
          thr = mulv(thr, albedo_effect0(m));
          thr0 = mulv(thr0, albedo_effect0(load_material(mat0 + 16u * mi)));
          const float tmx = smax(thr0.x, smax(thr0.y, thr0.z));
          if (!(tmx < 0.001f)) {
            const float rr = smin(st.rr_max, smax(st.rr_min, tmx));
            v.c.w = rr;
            if (!(depth >= st.rr_start && next01(rng) > rr)) {
              thr = divs(thr, rr);
              thr0 = divs(thr0, rr);
              next = depth + 1u < st.max_depth;
            }
          }
        }
        v.e = make_uint4(static_cast<uint32_t>(rng_at), static_cast<uint32_t>(rng_at >> 32), flags | (next ? kVfCont : 0u),
                         mi);
        if (next) {
          const V3 no = add(R.hp, mul(R.out, 0.002f));
          w.ray_o[p] = make_float4(no.x, no.y, no.z, 0.0f);
          w.ray_d[p] = make_float4(R.out.x, R.out.y, R.out.z, 0.0f);
          w.thr[p] = make_float4(thr.x, thr.y, thr.z, 0.0f);
          w.thr0[p] = make_float4(thr0.x, thr0.y, thr0.z, 0.0f);
          w.rng[p] = rng;
        }
      }
      rec[p] = v;
      if (!next) nrec[p] = depth + 1u;
      rad[p] = make_float4(r.x, r.y, r.z, 0.0f);
    }
    const uint32_t slot_n = warp_append(&ctl_word(w.counts, cur ^ 1u), next);
    if (next) qn[slot_n] = p;
    const uint32_t slot_s = warp_append(&ctl_word(w.counts, 2u + cur), shadow);
    if (shadow) {
      w.sh_path[slot_s] = p;
      w.sh_o[slot_s] = make_float4(R.q.origin.x, R.q.origin.y, R.q.origin.z, R.q.remain);
      w.sh_d[slot_s] = make_float4(R.q.dir.x, R.q.dir.y, R.q.dir.z, 0.0f);
      w.sh_c[slot_s] = make_float4(sh_c.x, sh_c.y, sh_c.z, 0.0f);
    }
  }
}

// adj_primal's hash of a path's decisions, from its records, into rad's w.
__global__ void __launch_bounds__(256) k_adj_sign(uint32_t n, const AdjRec* __restrict__ recs,
                                                  const uint32_t* __restrict__ nrec, float4* rad) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    uint64_t sig = 0u;
    const uint32_t k = nrec[j];
    for (uint32_t v = 0; v < k; ++v) {
      const AdjRec& r = recs[static_cast<size_t>(v) * n + j];
      const uint32_t flags = r.e.z;
      const uint64_t word = (flags & kVfMiss) ? 0xFFFFFFFFull
                                              : (static_cast<uint64_t>(__float_as_uint(r.b.w) + 1u) |
                                                 static_cast<uint64_t>(flags) << 32);
      sig = mix64(sig ^ word);
    }
    reinterpret_cast<float*>(rad + j)[3] = __uint_as_float(static_cast<uint32_t>(sig ^ (sig >> 32)));
  }
}

// Per pixel: film accumulation in sample order (non-finite samples dropped,
// optional firefly clamp), resolve, squared error (FP64) and the adjoint of
// each sample's radiance, 2 (img - target) / (3 W H) / count.
__global__ void __launch_bounds__(256) k_adj_loss(DevSettings st, uint32_t spp, const float4* rad, const float* target,
                                                  float* image, float4* adj, double* loss_part) {
  __shared__ double red[256];
  const uint32_t npx = st.width * st.height;
  double local = 0.0;
  const float scale = 2.0f / (3.0f * static_cast<float>(npx));
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npx; p += gridDim.x * blockDim.x) {
    float ax = 0.0f, ay = 0.0f, az = 0.0f;
    uint32_t cnt = 0u;
    for (uint32_t sl = 0; sl < spp; ++sl) {
      const float4 r = rad[static_cast<size_t>(sl) * npx + p];
      if (!(isfinite(r.x) && isfinite(r.y) && isfinite(r.z))) continue;
      float cx = r.x, cy = r.y, cz = r.z;
      if (st.firefly_clamp > 0.0f) {
        cx = smin(cx, st.firefly_clamp);
        cy = smin(cy, st.firefly_clamp);
        cz = smin(cz, st.firefly_clamp);
      }
      ax = ax + cx;
      ay = ay + cy;
      az = az + cz;
      ++cnt;
    }
    const float inv = 1.0f / static_cast<float>(cnt > 1u ? cnt : 1u);
    const float ix = ax * inv, iy = ay * inv, iz = az * inv;
    image[3 * p + 0] = ix;
    image[3 * p + 1] = iy;
    image[3 * p + 2] = iz;
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (target) {
      const float dx = ix - target[3 * p + 0], dy = iy - target[3 * p + 1], dz = iz - target[3 * p + 2];
      local += static_cast<double>(dx) * dx + static_cast<double>(dy) * dy + static_cast<double>(dz) * dz;
      g = make_float4(scale * dx * inv, scale * dy * inv, scale * dz * inv, 0.0f);
    }
    adj[p] = g;
  }
  red[threadIdx.x] = local;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (static_cast<int>(threadIdx.x) < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) loss_part[blockIdx.x] = red[0];
}

__global__ void k_adj_loss_final(const double* part, int n, double scale, double* loss) {
  __shared__ double red[256];
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += part[i];
  red[threadIdx.x] = v;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (static_cast<int>(threadIdx.x) < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = red[0] * scale;
}

// Gradient slots (sum, rounding error) per warp: a set for each group of eight lanes.
constexpr int kGradCopies = 4;

// Reverse sweep of one path.  `g` is dL/d(path radiance).  The warp runs the
// vertex loop in lockstep (k from the longest path's last vertex down) so the
// per-vertex gradients can be combined across lanes.
template <bool kParity>
__device__ __forceinline__ void adj_reverse(const DevScene& s, const DevSettings& st, const AdjRec* rec,
                                            uint32_t rec_stride, uint32_t nrec, bool lane_on, V3 g,
                                            float* stage, float2* warp_grad, uint32_t grad_stride) {
  const uint32_t kmax = __reduce_max_sync(0xffffffffu, lane_on ? nrec : 0u);
  const int lane = threadIdx.x & 31;
  V3 aT = mk(0.0f, 0.0f, 0.0f), aO = aT, aD = aT;
  for (int k = static_cast<int>(kmax) - 1; k >= 0; --k) {
    const bool act = lane_on && k < static_cast<int>(nrec);
    uint32_t mat = kMiss;
    float gv[kAdjParams] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (act) {
      const AdjRec r = rec[static_cast<size_t>(k) * rec_stride];
      const uint32_t flags = r.e.z;
      const V3 T = mk(r.c.x, r.c.y, r.c.z);
      if (flags & kVfMiss) {
        aT = mulv(g, s.env);
        aO = aD = mk(0.0f, 0.0f, 0.0f);
      } else {
        const uint32_t prim = __float_as_uint(r.b.w);
        const float4 sh = __ldg(s.shade + prim);
        const V3 gn = mk(sh.x, sh.y, sh.z);
        mat = r.e.w;
        const MaterialRec m = load_material(s.materials + 16u * mat);
        adj_vertex_vjp<kParity>(s, st, s.lights, static_cast<uint32_t>(k), mk(r.a.x, r.a.y, r.a.z),
                                mk(r.b.x, r.b.y, r.b.z), r.a.w, gn, m, T, r.c.w, flags,
                                static_cast<uint64_t>(r.e.x) | (static_cast<uint64_t>(r.e.y) << 32), g, aT, aO, aD, gv);
      }
    }
    // Add the lanes' gradients to the warp's slots: eight lanes (seven at work,
    // one per parameter) take every fourth source lane, each group of eight its
    // own copy of the slots, in a fixed order.  A tree over the lanes of one
    // material at a time cost 35 shuffles for each material of the warp
    // (0.41 ms a sweep of 524,288 paths against 0.36).  The slots carry their
    // rounding error along (Kahan): they take lanes one by one, so their
    // chains are longer than a tree's.
    __syncwarp();
    float4* mine = reinterpret_cast<float4*>(stage) + 2 * lane;
    mine[0] = make_float4(gv[0], gv[1], gv[2], gv[3]);
    mine[1] = make_float4(gv[4], gv[5], gv[6], __uint_as_float(mat));
    __syncwarp();
    const int copy = lane >> 3, param = lane & 7;
    if (param < static_cast<int>(kAdjParams)) {
      float2* slots = warp_grad + copy * grad_stride + param;
#pragma unroll
      for (int j = 0; j < 32; j += kGradCopies) {
        const float* src = stage + 8 * (j + copy);
        const uint32_t mj = __float_as_uint(src[7]);
        if (mj != kMiss) {
          float2& c = slots[mj * kAdjParams];
          const float y = src[param] - c.y, sum = c.x + y;
          c.y = isfinite(sum) ? (sum - c.x) - y : 0.0f;   // (an infinite sum has no error; inf - inf would be NaN)
          c.x = sum;
        }
      }
    }
  }
}

// The backward runs as two kernels per chunk of paths: the replay (the
// primal path again, with the traversal) writes every path's vertex records
// and its radiance adjoint to device memory, and the reverse sweep reads them.
// Split, each kernel's code is small enough for the instruction cache -- the
// fused kernel's warps waited on instruction fetch more than on anything else
// -- and each gets its own register budget.
// Records: vertex k of chunk path i at recs[k * count + i] (lanes of a warp
// touch consecutive records).
template <bool kParity>
__global__ void __launch_bounds__(128, 5) k_adj_replay(DevScene s, DevSettings st, const float* mat0,
                                                    uint32_t first_sample, int cap, const float4* adj,
                                                    const float* path_weight, uint64_t base, uint32_t count,
                                                    AdjRec* recs, float4* gout, uint32_t* err) {
  extern __shared__ int2 smem_dyn[];
  const TwoLevelStack stk = smem_stack_of(smem_dyn + threadIdx.x, static_cast<int>(blockDim.x), cap);
  const uint32_t npx = st.width * st.height;
  uint32_t local_err = 0u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint64_t j = base + i;
    const uint32_t sl = static_cast<uint32_t>(j / npx), p = static_cast<uint32_t>(j % npx);
    float4 a = adj[p];
    if (path_weight) {
      const float pw = path_weight[j];
      a = make_float4(a.x * pw, a.y * pw, a.z * pw, 0.0f);
    }
    V3 g = mk(0.0f, 0.0f, 0.0f);
    uint32_t nrec = 0u;
    if (a.x != 0.0f || a.y != 0.0f || a.z != 0.0f) {
      // The replayed radiance decides what the film would have dropped or
      // clamped (the replay may use other samples than the forward's).
      const float4 rv = adj_primal<kParity, true>(s, st, mat0, p % st.width, p / st.width, first_sample + sl, stk,
                                                  local_err, recs + i, nrec, count);
      const float fc = st.firefly_clamp;
      g = mk((fc > 0.0f && rv.x > fc) ? 0.0f : a.x, (fc > 0.0f && rv.y > fc) ? 0.0f : a.y,
             (fc > 0.0f && rv.z > fc) ? 0.0f : a.z);
      if (!(isfinite(rv.x) && isfinite(rv.y) && isfinite(rv.z))) nrec = 0u;
    }
    gout[i] = make_float4(g.x, g.y, g.z, __uint_as_float(nrec));
  }
  if (local_err) atomicOr(err, local_err);
}

// What the replay hands the reverse sweep, for paths the forward recorded
// (the same paths): each path's radiance adjoint (zero where the film
// dropped or clamped the sample, the path's weight applied) and its record
// count (0: nothing to sweep).
__global__ void __launch_bounds__(256) k_adj_gout(DevSettings st, const float4* adj, const float* path_weight,
                                                  const float4* rad, const uint32_t* nrec_fwd, uint32_t count,
                                                  float4* gout) {
  const uint32_t npx = st.width * st.height;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    float4 a = adj[i % npx];
    if (path_weight) {
      const float pw = path_weight[i];
      a = make_float4(a.x * pw, a.y * pw, a.z * pw, 0.0f);
    }
    V3 g = mk(0.0f, 0.0f, 0.0f);
    uint32_t nrec = 0u;
    if (a.x != 0.0f || a.y != 0.0f || a.z != 0.0f) {
      const float4 rv = rad[i];
      const float fc = st.firefly_clamp;
      g = mk((fc > 0.0f && rv.x > fc) ? 0.0f : a.x, (fc > 0.0f && rv.y > fc) ? 0.0f : a.y,
             (fc > 0.0f && rv.z > fc) ? 0.0f : a.z);
      nrec = (isfinite(rv.x) && isfinite(rv.y) && isfinite(rv.z)) ? nrec_fwd[i] : 0u;
    }
    gout[i] = make_float4(g.x, g.y, g.z, __uint_as_float(nrec));
  }
}

// The reverse sweep of one chunk: per-warp gradient slots in shared memory,
// then one partial per block, added to the partials of the earlier chunks
// (accumulate) in a fixed order, so the gradient is deterministic.
//
// Bound by instruction issue and fetch: a vertex is several hundred scalar
// instructions on about 14 of 32 lanes, its record 64 bytes.  Differentiating
// with seven-tangent dual numbers instead took 1.20 ms for 524,288 paths, two
// thirds of its stalls waiting for instructions; the vector-Jacobian product
// 0.41 ms, with the slots added through shared memory 0.36 and with their
// rounding errors carried along 0.38.  Four blocks (128 registers) 0.36 ms,
// five (96) 0.40, six (80) 0.42.
template <bool kParity>
__global__ void __launch_bounds__(128, 4) k_adj_reverse(DevScene s, DevSettings st, uint32_t count,
                                                     const AdjRec* recs, const float4* gout, float* grad_part,
                                                     int accumulate) {
  extern __shared__ float4 smem_reverse[];   // per warp 32 x 8 floats of staging, then the slots
  float* smem = reinterpret_cast<float*>(smem_reverse);
  const int warps = blockDim.x >> 5;
  const uint32_t stride = s.material_count * kAdjParams;
  float* stage = smem + (threadIdx.x >> 5) * 256;
  float2* grads = reinterpret_cast<float2*>(smem + warps * 256);
  const int slots = warps * kGradCopies;
  for (uint32_t i = threadIdx.x; i < stride * slots; i += blockDim.x) grads[i] = make_float2(0.0f, 0.0f);
  __syncthreads();
  float2* warp_grad = grads + (threadIdx.x >> 5) * kGradCopies * stride;
  for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    V3 g = mk(0.0f, 0.0f, 0.0f);
    uint32_t nrec = 0u;
    if (i < count) {
      const float4 gv = gout[i];
      g = mk(gv.x, gv.y, gv.z);
      nrec = __float_as_uint(gv.w);
    }
    adj_reverse<kParity>(s, st, recs + (i < count ? i : 0u), count, nrec, nrec != 0u, g, stage,
                         warp_grad, stride);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < stride; i += blockDim.x) {
    double sum = 0.0;
    for (int w = 0; w < slots; ++w) {
      const float2 c = grads[w * stride + i];
      sum += static_cast<double>(c.x) - c.y;
    }
    const float v = static_cast<float>(sum);
    float* dst = grad_part + static_cast<size_t>(blockIdx.x) * stride + i;
    *dst = accumulate ? *dst + v : v;
  }
}

__global__ void k_adj_grad_reduce(const float* part, int blocks, uint32_t stride, float* grad) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < stride; i += gridDim.x * blockDim.x) {
    double v = 0.0;
    for (int b = 0; b < blocks; ++b) v += part[static_cast<size_t>(b) * stride + i];
    grad[i] = static_cast<float>(v);
  }
}

}  // namespace

size_t AdjForwardSmem(int block, int stack_cap) { return static_cast<size_t>(block) * stack_cap * sizeof(int2); }

size_t AdjBackwardSmem(int block, int stack_cap, uint32_t materials) {
  return std::max(AdjForwardSmem(block, stack_cap), AdjReverseSmem(block, materials));
}

size_t AdjReverseSmem(int block, uint32_t materials) {
  return static_cast<size_t>(block / 32) * (256 + 2 * kGradCopies * materials * kAdjParams) * sizeof(float);
}

int AdjBlocksPerSm(AdjKernel k, int block, size_t smem, bool parity) {
  int n = 0;
  switch (k) {
    case AdjKernel::kForward:
      if (parity) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_forward<true, false>, block, smem);
      else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_forward<false, false>, block, smem);
      break;
    case AdjKernel::kReplay:
      if (parity) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_replay<true>, block, smem);
      else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_replay<false>, block, smem);
      break;
    case AdjKernel::kReverse:
      if (parity) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_reverse<true>, block, smem);
      else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_reverse<false>, block, smem);
      break;
  }
  return n > 0 ? n : 1;
}

cudaError_t ConfigureAdjSmem() {
  cudaError_t e;
  if ((e = allow_full_smem(k_adj_forward<true, false>))) return e;
  if ((e = allow_full_smem(k_adj_forward<false, false>))) return e;
  if ((e = allow_full_smem(k_adj_forward<true, true>))) return e;
  if ((e = allow_full_smem(k_adj_forward<false, true>))) return e;
  if ((e = allow_full_smem(k_adj_replay<true>))) return e;
  if ((e = allow_full_smem(k_adj_replay<false>))) return e;
  if ((e = allow_full_smem(k_adj_reverse<true>))) return e;
  return allow_full_smem(k_adj_reverse<false>);
}

cudaError_t LaunchAdjForward(const DevScene& s, const DevSettings& st, const float* mat0, const AdjLaunch& l,
                             float4* rad, uint32_t* err, float4* recs, uint32_t* nrec) {
  const size_t smem = AdjForwardSmem(l.block, l.stack_cap);
  AdjRec* r = reinterpret_cast<AdjRec*>(recs);
  const bool rec = recs != nullptr && nrec != nullptr;
#define VKPTC_FWD(P, R) \
  k_adj_forward<P, R><<<l.grid, l.block, smem, l.stream>>>(s, st, mat0, l.spp, l.first_sample, l.stack_cap, rad, r, nrec, err)
  if (l.parity && rec) VKPTC_FWD(true, true);
  else if (l.parity) VKPTC_FWD(true, false);
  else if (rec) VKPTC_FWD(false, true);
  else VKPTC_FWD(false, false);
#undef VKPTC_FWD
  return cudaGetLastError();
}

cudaError_t ConfigureAdjTraceSmem() { return allow_full_smem(k_adj_trace); }

cudaError_t LaunchAdjRecord(const DevScene& s, const DevSettings& st, const float* mat0, const AdjWaveLaunch& l,
                            const AdjWave& w, float4* rad, float4* recs, uint32_t* nrec, uint32_t* err) {
  const uint32_t n = st.width * st.height * l.spp;
  AdjRec* r = reinterpret_cast<AdjRec*>(recs);
  const size_t smem = static_cast<size_t>(l.block) * l.smem_entries * sizeof(int2);
  constexpr int kShadeBlock = 128;   // k_adj_shade's bound
  const int shade_grid = std::max(1, l.grid * l.block / kShadeBlock);
  if (l.parity) k_adj_raygen<true><<<l.grid, l.block, 0, l.stream>>>(s, st, n, l.first_sample, w, rad);
  else k_adj_raygen<false><<<l.grid, l.block, 0, l.stream>>>(s, st, n, l.first_sample, w, rad);
  for (uint32_t depth = 0; depth < st.max_depth; ++depth) {
    const uint32_t* q = w.q[depth & 1u];
    uint32_t* qn = w.q[(depth & 1u) ^ 1u];
    AdjRec* rec = r + static_cast<size_t>(depth) * n;
    k_adj_trace<<<l.grid, l.block, smem, l.stream>>>(s, w, q, depth, rad, depth > 0u ? rec - n : rec, l.smem_entries,
                                                     l.spill, l.stack_cap, l.steps, err);
    if (l.parity) k_adj_shade<true><<<shade_grid, kShadeBlock, 0, l.stream>>>(s, st, mat0, w, q, qn, depth, rad, rec, nrec);
    else k_adj_shade<false><<<shade_grid, kShadeBlock, 0, l.stream>>>(s, st, mat0, w, q, qn, depth, rad, rec, nrec);
  }
  k_adj_sign<<<l.grid, l.block, 0, l.stream>>>(n, r, nrec, rad);
  return cudaGetLastError();
}

cudaError_t LaunchAdjLoss(const DevSettings& st, uint32_t spp, const float4* rad, const float* target, float* image,
                          float4* adj, double* loss_part, double* loss, int grid, cudaStream_t stream) {
  k_adj_loss<<<grid, 256, 0, stream>>>(st, spp, rad, target, image, adj, loss_part);
  const double npx = static_cast<double>(st.width) * st.height;
  k_adj_loss_final<<<1, 256, 0, stream>>>(loss_part, grid, 1.0 / (3.0 * npx), loss);
  return cudaGetLastError();
}

cudaError_t LaunchAdjBackward(const DevScene& s, const DevSettings& st, const float* mat0, const AdjLaunch& l,
                              const float4* adj, const float* path_weight, float4* recs, float4* gout,
                              float* grad_part, float* grad, uint32_t* err, const float4* fwd_rad,
                              const uint32_t* fwd_nrec) {
  const size_t smem_replay = AdjForwardSmem(l.block, l.stack_cap);
  const size_t smem_rev = AdjReverseSmem(l.block, s.material_count);
  const uint64_t n = static_cast<uint64_t>(st.width) * st.height * l.spp;
  AdjRec* r = reinterpret_cast<AdjRec*>(recs);
  if (fwd_rad != nullptr && fwd_nrec != nullptr && n <= kAdjChunkPaths) {
    // the forward recorded these paths: no replay
    const uint32_t count = static_cast<uint32_t>(n);
    k_adj_gout<<<static_cast<int>(std::min<uint64_t>(4096, (n + 255) / 256)), 256, 0, l.stream>>>(
        st, adj, path_weight, fwd_rad, fwd_nrec, count, gout);
    if (l.parity) k_adj_reverse<true><<<l.grid_reverse, l.block, smem_rev, l.stream>>>(s, st, count, r, gout, grad_part, 0);
    else k_adj_reverse<false><<<l.grid_reverse, l.block, smem_rev, l.stream>>>(s, st, count, r, gout, grad_part, 0);
    const uint32_t stride = s.material_count * kAdjParams;
    k_adj_grad_reduce<<<(stride + 127) / 128, 128, 0, l.stream>>>(grad_part, l.grid_reverse, stride, grad);
    return cudaGetLastError();
  }
  for (uint64_t base = 0; base < n; base += kAdjChunkPaths) {
    const uint32_t count = static_cast<uint32_t>(std::min<uint64_t>(kAdjChunkPaths, n - base));
    const int acc = base > 0 ? 1 : 0;
    if (l.parity) {
      k_adj_replay<true><<<l.grid, l.block, smem_replay, l.stream>>>(s, st, mat0, l.first_sample, l.stack_cap, adj,
                                                                   path_weight, base, count, r, gout, err);
      k_adj_reverse<true><<<l.grid_reverse, l.block, smem_rev, l.stream>>>(s, st, count, r, gout, grad_part, acc);
    } else {
      k_adj_replay<false><<<l.grid, l.block, smem_replay, l.stream>>>(s, st, mat0, l.first_sample, l.stack_cap, adj,
                                                                    path_weight, base, count, r, gout, err);
      k_adj_reverse<false><<<l.grid_reverse, l.block, smem_rev, l.stream>>>(s, st, count, r, gout, grad_part, acc);
    }
  }
  const uint32_t stride = s.material_count * kAdjParams;
  k_adj_grad_reduce<<<(stride + 127) / 128, 128, 0, l.stream>>>(grad_part, l.grid_reverse, stride, grad);
  return cudaGetLastError();
}

}  // namespace vkptc
