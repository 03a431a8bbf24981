// adjoint.cuh -- differentiable path tracing: the per-vertex integrator math
// (adj_vertex) and its vector-Jacobian product (adj_vertex_vjp), which the
// reverse sweep pulls the adjoints of a vertex's results through.
//
// There is no counterpart in the reference (its tracer has no derivative
// path).  The primal follows the reference's trace loop
// (src/pathtracer/ScalarCpuPathTracer.cpp:1148-1289), sample_direct_light
// (:1022-1118) and sample_phong_lobe (:996-1020) in the same operation order
// as shade_bounce / nee_setup / sample_phong, for the materials the adjoint
// supports: Lambertian and Phong-lobe glossy (models 0, 1, 3; no metal,
// mirror, clear coat or transmission), optionally emissive.
//
// Estimator differentiated (it is the one the FP64 CPU adjoint restates):
//   * directions are reparameterized: a Phong-lobe direction is a function of
//     its two uniforms, the reflected direction and the exponent, so it moves
//     with the roughness and with the incoming direction; a hemisphere
//     direction depends on nothing differentiable;
//   * the Russian-roulette survival probability is held constant (detached):
//     throughput divides by it, but no derivative flows through it;
//   * every discrete decision (hit primitive, visibility, lobe fallback,
//     frame choice, termination) is taken from the primal replay, so
//     visibility-boundary terms are excluded.
#pragma once

#include "integrator.cuh"

namespace vkptc {

constexpr uint32_t kAdjMaxDepth = 8u;     // vertices recorded per path
constexpr uint32_t kAdjParams = 7u;       // per material: albedo rgb, roughness, emission rgb
constexpr uint32_t kAdjMaxMaterials = 64u;

// Vertex flags recorded by the primal replay.
enum : uint32_t {
  kVfEntering = 1u << 0,    // the ray arrived from the geometric normal's side
  kVfNeeValid = 1u << 1,    // sample_direct_light produced a candidate
  kVfNeeVis = 1u << 2,      // ... and its contribution was added
  kVfFrameAlt = 1u << 3,    // Phong frame built around (0,1,0)
  kVfReflected = 1u << 4,   // Phong direction mirrored about the normal
  kVfHemi = 1u << 5,        // ... and replaced by a hemisphere direction
  kVfCont = 1u << 6,        // the path continues to the next vertex
  kVfMiss = 1u << 7,        // the ray left the scene (environment term)
};

// ------------------------------------------------------------- vertex math
// Emission MIS weight's light pdf (light_pdf_for_direction,
// ScalarCpuPathTracer.cpp:1120-1138) over a generic origin/direction.
__device__ __forceinline__ float adj_light_pdf(const DevScene& s, const float* lights, V3 p, V3 dir) {
  float total = 0.0f;
  if (s.light_count == 0u) return total;
  const float inv_n = 1.0f / static_cast<float>(s.light_count);
  for (uint32_t k = 0; k < s.light_count; ++k) {
    const V3 tl = sub(ld3(lights + 16u * k), p);
    const float dist = sqrtf(dot(tl, tl));
    if (dist < kEps) continue;
    if (dot(divs(tl, dist), dir) > 0.9999f) total = total + inv_n / (dist * dist + kEps);
  }
  return total;
}

__device__ __forceinline__ float adj_mis(float a, float b) {
  const float a2 = a * a, b2 = b * b, den = a2 + b2;
  if (den <= 0.0f) return 1.0f;
  return a2 / den;
}

__device__ __forceinline__ float adj_spot(const float* L, V3 from_light) {
  const float inner = L[11], outer = L[12];
  if (inner <= -0.999f) return 1.0f;
  const float cone = dot(unit(from_light), unit(ld3(L + 8)));
  if (cone <= outer) return 0.0f;
  if (cone >= inner || inner <= outer) return 1.0f;
  const float t = sclamp((cone - outer) / (inner - outer), 0.0f, 1.0f);
  return t * t * (3.0f - 2.0f * t);
}

// Next-event estimate at `p` (normal n, material m, viewing direction view):
// radiance R (before the MIS weight and the throughput) and the shadow segment.
struct AdjNee {
  V3 radiance, origin, dir;
  float remain;
};

// The sampled point of the chosen light; returns the light's record.
template <bool kParity>
__device__ __forceinline__ const float* adj_pick_light(const DevScene& s, const float* lights, uint64_t& rng, V3& lp) {
  const uint32_t nl = s.light_count;
  uint32_t pick = static_cast<uint32_t>(next01(rng) * static_cast<float>(nl));
  if (pick > nl - 1u) pick = nl - 1u;
  const float* L = lights + 16u * pick;
  lp = ld3(L);
  const float radius = L[7];
  if (radius > 1.0e-5f) {
    const float uz = 1.0f - 2.0f * next01(rng);
    const float r = sqrtf(smax(0.0f, 1.0f - uz * uz));
    const float phi = 6.28318530718f * next01(rng);
    lp = add(lp, mul(mk(r * t_cos<kParity>(phi), uz, r * t_sin<kParity>(phi)), radius));
  }
  return L;
}

template <bool kParity>
__device__ __forceinline__ bool adj_nee(const DevScene& s, const float* lights, V3 p, V3 n, const MaterialRec& m,
                                        float rough, V3 view, uint64_t& rng, uint32_t& flags, AdjNee& q) {
  const uint32_t nl = s.light_count;
  if (nl == 0u) return false;
  V3 lp;
  const float* L = adj_pick_light<kParity>(s, lights, rng, lp);
  const V3 tl = sub(lp, p);
  const float d2 = dot(tl, tl);
  const float dist = sqrtf(d2);
  if (dist < kEps) return false;
  const V3 ldir = divs(tl, dist);
  const float cth = dot(n, ldir);
  if (cth <= 0.0f) return false;
  const float sf = adj_spot(L, neg(ldir));
  if (sf <= 0.0f) return false;
  const V3 alb = albedo_effect0(m);
  const V3 irr = mul(ld3(L + 3), (L[6] * sf) / (d2 + kEps));
  const float fnl = static_cast<float>(nl);
  // Diffuse term (no mirror or transmissive material reaches here).
  V3 acc = mul(mul(mulv(mul(alb, kInvPi), irr), cth), fnl);
  if (rough < 0.65f) {
    const V3 hv = unit(add(ldir, unit(view)));
    const float er = smax(0.025f, rough * 1.0f);
    const float a2 = er * er;
    const float pw = sclamp(2.0f / smax(0.0005f, a2 * a2) - 2.0f, 4.0f, 96.0f);
    const float spec = t_pow<kParity>(smax(0.0f, dot(n, hv)), pw);
    const float ss = clamp01((1.0f - rough) * 0.8f + m.metallic * 0.45f + m.clearcoat * 0.35f + 0.0f + 0.0f);
    const V3 tint = add(mul(mk(1.0f, 1.0f, 1.0f), 0.88f), mul(alb, 0.12f));
    acc = add(acc, mul(mulv(tint, irr), spec * cth * fnl * smax(0.15f, ss)));
  }
  flags |= kVfNeeValid;
  q.radiance = acc;
  q.origin = add(p, mul(n, 0.002f));
  q.dir = ldir;
  q.remain = dist - 0.004f;
  return true;
}

// Phong-lobe direction around refl (sample_phong_lobe, :996-1020).
template <bool kParity>
__device__ __forceinline__ V3 adj_phong(uint64_t& rng, V3 refl, float ex, V3 n, uint32_t& flags) {
  const float u1 = next01(rng);
  const float u2 = next01(rng);
  const float ct = t_pow<kParity>(smax(0.0f, u1), 1.0f / (ex + 1.0f));
  const float sn = sqrtf(smax(0.0f, 1.0f - ct * ct));
  const float phi = 2.0f * kPi * u2;
  const bool alt = !(fabsf(refl.z) < 0.999f);
  if (alt) flags |= kVfFrameAlt;
  const V3 ref = alt ? mk(0.0f, 1.0f, 0.0f) : mk(0.0f, 0.0f, 1.0f);
  const V3 t = unit(cross(ref, refl));
  const V3 b = cross(refl, t);
  V3 out = unit(add(add(mul(t, sn * t_cos<kParity>(phi)), mul(b, sn * t_sin<kParity>(phi))), mul(refl, ct)));
  if (dot(out, n) <= 0.0f) {
    flags |= kVfReflected;
    out = sub(out, mul(n, 2.0f * dot(out, n)));
    if (dot(out, n) <= 0.0f) {
      flags |= kVfHemi;
      return sample_hemisphere<kParity>(rng, n);
    }
  }
  return out;
}

// What one vertex contributes.
struct AdjVertex {
  V3 hp;
  float w_e;          // emission weight: (T * Le) * w_e is added
  bool nee;           // NEE candidate present (kVfNeeValid)
  AdjNee q;
  float w_n;          // NEE MIS weight: (T * R) * w_n is added when visible
  V3 out;             // next direction (valid when the material scattered)
  bool scattered;     // a direction was sampled above the surface
};

// Hit shading of one vertex (without the visibility test and the
// throughput update, which the caller does).
template <bool kParity>
__device__ __forceinline__ void adj_vertex(const DevScene& s, const DevSettings& st, const float* lights,
                                           uint32_t depth, V3 o, V3 d, float ht, V3 gn, const MaterialRec& m,
                                           float rough, uint64_t& rng, uint32_t& flags, AdjVertex& R) {
  R.hp = add(o, mul(d, ht));
  const bool entering = dot(d, gn) < 0.0f;
  if (entering) flags |= kVfEntering;
  const V3 nv = entering ? gn : neg(gn);
  const bool emissive_any = m.emissive.x > 0.0f || m.emissive.y > 0.0f || m.emissive.z > 0.0f;
  const bool emissive_model = m.model == 1u || emissive_any;
  const bool diffuse = rough >= 0.999f;

  if (!st.enable_nee || depth == 0u) {
    R.w_e = 1.0f;
  } else if (st.enable_mis && emissive_model) {
    const float bp = smax(0.0f, dot(nv, neg(d))) * kInvPi;
    const float lpdf = adj_light_pdf(s, lights, o, d);
    R.w_e = adj_mis(bp, lpdf);
  } else {
    R.w_e = 0.0f;
  }

  R.nee = false;
  if (st.enable_nee && depth < st.max_depth - 1u) {
    R.nee = adj_nee<kParity>(s, lights, R.hp, nv, m, rough, neg(d), rng, flags, R.q);
    if (R.nee) {
      if (st.enable_mis) {
        const V3 ld = unit(sub(ld3(lights), R.hp));
        const float bp = smax(0.0f, dot(nv, ld)) * kInvPi;
        const float lpdf = 1.0f / static_cast<float>(s.light_count);
        R.w_n = adj_mis(lpdf, bp);
      } else {
        R.w_n = 1.0f;
      }
    }
  }

  const V3 refl = sub(d, mul(nv, 2.0f * dot(nv, d)));
  if (diffuse) {
    R.out = sample_hemisphere<kParity>(rng, nv);
  } else {
    const float er = smax(0.025f, rough * 1.0f * 1.0f);
    const float a2 = er * er;
    const float ex = smax(0.0f, 2.0f / (a2 * a2) - 2.0f);
    R.out = adj_phong<kParity>(rng, refl, ex, nv, flags);
  }
  R.scattered = !(dot(R.out, nv) <= 0.0f);
}

// ------------------------------------------------- vector-Jacobian products
// u = v / |v| (unit's constant fallback below kEps): the adjoint of v.
__device__ __forceinline__ V3 vjp_unit(V3 u, float len, V3 au) {
  if (len <= kEps) return mk(0.0f, 0.0f, 0.0f);
  return mul(sub(au, mul(u, dot(u, au))), 1.0f / len);
}
__device__ __forceinline__ V3 unit_len(V3 v, float& len) {
  len = sqrtf(dot(v, v));
  return len <= kEps ? mk(0.0f, 1.0f, 0.0f) : divs(v, len);
}
// w = a^2 / (a^2 + b^2) (1 where the denominator vanishes) with dw/da, dw/db.
__device__ __forceinline__ float mis_grad(float a, float b, float& da, float& db) {
  const float a2 = a * a, b2 = b * b, den = a2 + b2;
  da = db = 0.0f;
  if (den <= 0.0f) return 1.0f;
  const float inv = 1.0f / den, w = a2 / den;
  da = 2.0f * a * (b2 * inv) * inv;
  db = -2.0f * b * w * inv;
  return w;
}

// Adjoints at one vertex.  In: g = dL/d(path radiance), the vertex's record
// (incoming ray o, d, hit distance th, throughput T, Russian-roulette factor,
// flags, generator state) and the adjoints aT, aO, aD of what the path
// carries to the next vertex.  Out: the same adjoints for what it carried
// into this one, and gv = the material's gradient.
//
// Each of the three contributions (emission, next event, scattered ray) is
// recomputed and differentiated backwards where it stands, in scalars: the
// vertex has about ten outputs with an adjoint (the next ray, two weights,
// a radiance) but only their one weighted sum is differentiated, so the
// reverse direction needs one adjoint per intermediate where seven-tangent
// dual numbers carried seven.  The next event is recomputed only where it was
// visible, the scattered direction only where the path went on.  Decisions
// come from the record's flags.
template <bool kParity>
__device__ __forceinline__ void adj_vertex_vjp(const DevScene& s, const DevSettings& st, const float* lights,
                                               uint32_t depth, V3 o, V3 d, float th, V3 gn, const MaterialRec& m,
                                               V3 T, float rr, uint32_t flags, uint64_t rng, V3 g, V3& aT, V3& aO,
                                               V3& aD, float (&gv)[kAdjParams]) {
  const float rough = clamp01(m.roughness);
  const V3 hp = add(o, mul(d, th));
  const V3 nv = (flags & kVfEntering) ? gn : neg(gn);
  const V3 alb = albedo_effect0(m);
  const V3 amask = mk((m.albedo.x > 0.0f && m.albedo.x < 1.5f) ? 1.0f : 0.0f,
                      (m.albedo.y > 0.0f && m.albedo.y < 1.5f) ? 1.0f : 0.0f,
                      (m.albedo.z > 0.0f && m.albedo.z < 1.5f) ? 1.0f : 0.0f);
  const V3 q = mulv(g, T);
  V3 a_o = mk(0.0f, 0.0f, 0.0f), a_d = a_o, a_hp = a_o, galb = a_o;
  float a_rough = 0.0f;

  // Emission: (T * Le) * w_e.
  float we = 0.0f;
  const bool emissive_any = m.emissive.x > 0.0f || m.emissive.y > 0.0f || m.emissive.z > 0.0f;
  if (!st.enable_nee || depth == 0u) {
    we = 1.0f;
  } else if (st.enable_mis && (m.model == 1u || emissive_any)) {
    const float x = dot(nv, neg(d));
    const float bp = smax(0.0f, x) * kInvPi;
    float lpdf = 0.0f;
    V3 dl = mk(0.0f, 0.0f, 0.0f);   // d lpdf / d o
    const float inv_n = 1.0f / static_cast<float>(s.light_count);
    for (uint32_t k = 0; k < s.light_count; ++k) {
      const V3 tl = sub(ld3(lights + 16u * k), o);
      const float dist = sqrtf(dot(tl, tl));
      if (dist < kEps) continue;
      if (dot(divs(tl, dist), d) > 0.9999f) {
        const float den = dist * dist + kEps, pdf = inv_n / den;
        lpdf = lpdf + pdf;
        dl = add(dl, mul(tl, 2.0f * pdf / den));
      }
    }
    float da, db;
    we = mis_grad(bp, lpdf, da, db);
    const float se = q.x * m.emissive.x + q.y * m.emissive.y + q.z * m.emissive.z;
    if (0.0f < x) a_d = mul(nv, -(se * da * kInvPi));
    a_o = mul(dl, se * db);
  }
  gv[4] = q.x * we;
  gv[5] = q.y * we;
  gv[6] = q.z * we;
  V3 aTk = mul(mulv(g, m.emissive), we);

  // Next event: (T * R) * w_n where it was added.
  if (st.enable_nee && depth < st.max_depth - 1u && s.light_count != 0u) {
    V3 lp;
    const float* L = adj_pick_light<kParity>(s, lights, rng, lp);
    if ((flags & (kVfNeeValid | kVfNeeVis)) == (kVfNeeValid | kVfNeeVis)) {
      const float fnl = static_cast<float>(s.light_count);
      float wn = 1.0f, dwn = 0.0f, len0 = 0.0f, y = 0.0f;
      V3 l0 = mk(0.0f, 0.0f, 0.0f);
      if (st.enable_mis) {
        l0 = unit_len(sub(ld3(lights), hp), len0);
        y = dot(nv, l0);
        float da;
        wn = mis_grad(1.0f / fnl, smax(0.0f, y) * kInvPi, da, dwn);
      }
      const V3 tl = sub(lp, hp);
      const float d2 = dot(tl, tl), dist = sqrtf(d2);
      const V3 ldir = divs(tl, dist);
      const float cth = dot(nv, ldir);
      const V3 Le = ld3(L + 3);
      const float power = L[6], inner = L[11], outer = L[12];
      // spot falloff
      float sf = 1.0f, dsf = 0.0f, flen = 0.0f;
      V3 fu = mk(0.0f, 0.0f, 0.0f), axis = fu;
      if (inner > -0.999f) {
        fu = unit_len(neg(ldir), flen);
        axis = unit(ld3(L + 8));
        const float cone = dot(fu, axis);
        if (cone <= outer) {
          sf = 0.0f;
        } else if (!(cone >= inner || inner <= outer)) {
          const float w = inner - outer, t = (cone - outer) / w;
          sf = t * t * (3.0f - 2.0f * t);
          dsf = 6.0f * t * (1.0f - t) / w;
        }
      }
      const float den = d2 + kEps, k = (power * sf) / den;   // irradiance = Le * k
      // R_i = Le_i k (alb_i/pi cth n + tint_i spec_w); sums over the channels
      // weighted with their adjoints: c for the diffuse, e for the glossy part.
      const V3 qle = mulv(q, Le);
      const float kd = cth * fnl * kInvPi;
      float c = qle.x * alb.x + qle.y * alb.y + qle.z * alb.z, e = 0.0f, spec_w = 0.0f;
      V3 a_ldir = mk(0.0f, 0.0f, 0.0f);
      float a_cth = wn * k * c * fnl * kInvPi;
      V3 rad = mul(alb, k * kd);
      if (rough < 0.65f) {
        float lv, lh;
        const V3 vu = unit_len(neg(d), lv);
        const V3 hv = unit_len(add(ldir, vu), lh);
        const float x = dot(nv, hv), er = smax(0.025f, rough), a2 = er * er, a4 = a2 * a2;
        const float z = smax(0.0005f, a4), pw0 = 2.0f / z - 2.0f, pw = sclamp(pw0, 4.0f, 96.0f);
        const float spec = t_pow<kParity>(smax(0.0f, x), pw);
        const float ss0 = (1.0f - rough) * 0.8f + m.metallic * 0.45f + m.clearcoat * 0.35f;
        const float ss = clamp01(ss0), ssw = smax(0.15f, ss);
        const float ws = cth * fnl * ssw;
        spec_w = spec * ws;
        const V3 tint = mk(0.88f + 0.12f * alb.x, 0.88f + 0.12f * alb.y, 0.88f + 0.12f * alb.z);
        e = qle.x * tint.x + qle.y * tint.y + qle.z * tint.z;
        rad = add(rad, mul(tint, k * spec_w));
        const float a_w = wn * k * e;     // adjoint of spec_w
        a_cth += a_w * spec * fnl * ssw;
        if (0.15f < ss && 0.0f < ss0 && ss0 < 1.0f) a_rough -= 0.8f * (a_w * spec * cth * fnl);
        if (x > 0.0f) {
          const float a_spec = a_w * ws;
          const V3 a_h = vjp_unit(hv, lh, mul(nv, a_spec * (spec * pw / x)));
          a_ldir = a_h;
          a_d = sub(a_d, vjp_unit(vu, lv, a_h));
          if (pw0 >= 4.0f && pw0 <= 96.0f && 0.0005f < a4 && 0.025f < rough)
            a_rough -= a_spec * spec * logf(x) * (8.0f * er * a2 / (z * z));
        }
      }
      rad = mulv(rad, Le);
      const float a_k = wn * (c * kd + e * spec_w);
      a_ldir = add(a_ldir, mul(nv, a_cth));
      if (dsf != 0.0f) a_ldir = sub(a_ldir, vjp_unit(fu, flen, mul(axis, a_k * power / den * dsf)));
      V3 a_tl = vjp_unit(ldir, dist, a_ldir);
      a_tl = sub(a_tl, mul(tl, 2.0f * (a_k * k / den)));
      a_hp = sub(a_hp, a_tl);
      const float sr = q.x * rad.x + q.y * rad.y + q.z * rad.z;
      if (0.0f < y) a_hp = sub(a_hp, vjp_unit(l0, len0, mul(nv, sr * dwn * kInvPi)));
      const float pa = wn * k * (kd + 0.12f * spec_w);
      galb = mulv(mul(qle, pa), amask);
      aTk = add(aTk, mul(mulv(g, rad), wn));
    }
  }

  // Throughput T' = T * albedo / rr (rr held constant) and the next ray.
  if (flags & kVfCont) {
    const float inv_rr = 1.0f / rr;
    aTk = add(aTk, mul(mulv(aT, alb), inv_rr));
    galb = add(galb, mulv(mul(mulv(aT, T), inv_rr), amask));
    a_hp = add(a_hp, aO);
    if (rough < 0.999f && !(flags & kVfHemi)) {
      const V3 refl = sub(d, mul(nv, 2.0f * dot(nv, d)));
      const float er = smax(0.025f, rough), a2 = er * er, ex0 = 2.0f / (a2 * a2) - 2.0f;
      const float u1 = smax(0.0f, next01(rng)), u2 = next01(rng);
      const float yexp = 1.0f / (smax(0.0f, ex0) + 1.0f);
      const float ct = t_pow<kParity>(u1, yexp);
      const float arg = 1.0f - ct * ct, sn = sqrtf(smax(0.0f, arg));
      const float phi = 2.0f * kPi * u2, cp = t_cos<kParity>(phi), sp = t_sin<kParity>(phi);
      const V3 ref = (flags & kVfFrameAlt) ? mk(0.0f, 1.0f, 0.0f) : mk(0.0f, 0.0f, 1.0f);
      float lt, lw;
      const V3 t = unit_len(cross(ref, refl), lt);
      const V3 b = cross(refl, t);
      const V3 w = unit_len(add(add(mul(t, sn * cp), mul(b, sn * sp)), mul(refl, ct)), lw);
      V3 a_out = add(aD, mul(aO, 0.002f));
      if (flags & kVfReflected) a_out = sub(a_out, mul(nv, 2.0f * dot(nv, a_out)));
      const V3 a_w = vjp_unit(w, lw, a_out);
      const V3 a_b = mul(a_w, sn * sp);
      const V3 a_t = add(mul(a_w, sn * cp), cross(a_b, refl));
      V3 a_refl = add(add(mul(a_w, ct), cross(t, a_b)), cross(vjp_unit(t, lt, a_t), ref));
      float a_ct = dot(refl, a_w);
      if (0.0f < arg) a_ct -= (cp * dot(t, a_w) + sp * dot(b, a_w)) * ct / sn;
      // ct = u1^y, y = 1 / (ex + 1), ex = 2 / er^4 - 2
      if (u1 > 0.0f && 0.0f < ex0 && 0.025f < rough)
        a_rough += a_ct * ct * logf(u1) * yexp * yexp * (8.0f / (a2 * a2 * er));
      a_d = add(a_d, sub(a_refl, mul(nv, 2.0f * dot(nv, a_refl))));
    }
  }

  // hp = o + d t on the hit triangle's plane, t = (v0 - o).n / (d.n).
  a_o = add(a_o, a_hp);
  a_d = add(a_d, mul(a_hp, th));
  const float dn = dot(d, gn);
  if (dn != 0.0f) {
    const float a_t = dot(d, a_hp) / dn;
    a_o = sub(a_o, mul(gn, a_t));
    a_d = sub(a_d, mul(gn, th * a_t));
  }
  gv[0] = galb.x;
  gv[1] = galb.y;
  gv[2] = galb.z;
  gv[3] = (m.roughness > 0.0f && m.roughness < 1.0f) ? a_rough : 0.0f;
  aT = aTk;
  aO = a_o;
  aD = a_d;
}

}  // namespace vkptc
