// yc_shade.cuh -- per-vertex shading of the wavefront path tracer (device side).
//
// Each function performs the arithmetic of its kernels/legacy/udpt.cl counterpart in
// the same FP32 operation order (cited per function), with the ym:: built-ins, so a
// path consumes the same random numbers and produces the same bits as the CPU oracle.
// Points carry w = 1 and directions w = 0, as in the reference's float4 values; the
// w lanes are kept because the four-lane dot products and the NaN test of the final
// colour see them.
#pragma once

#include "../ym_math.h"
#include "yc_scene.h"

namespace yc {

using ym::f4;

constexpr float PI_F = 3.14159265359f;
constexpr float INV_PI_F = 0.31830988618f;
constexpr float EPS_F = 0.0001f;
// largest float f with (double)f <= 0.0001: |DdotN| > 0.0001 (udpt.cl:247, compared in
// double) holds exactly when |DdotN| > this value
constexpr uint32_t LIGHT_DDOTN_BITS = 0x38D1B717u;

__device__ __forceinline__ f4 ld4(const yc_float4& v) { return ym::mk(v.x, v.y, v.z, v.w); }
__device__ __forceinline__ f4 f4of(float4 v) { return ym::mk(v.x, v.y, v.z, v.w); }
__device__ __forceinline__ float draw(uint32_t& seed) { seed = ym::xor_shift(seed); return ym::u01(seed); }

// What a step of a path sends: one closest-hit ray, or none (the path then waits for segments), and
// segments (segment s: EMIT_SEG0 << s)
enum : int { EMIT_CLOSEST = 1, EMIT_WAIT = 2, EMIT = 3, EMIT_SEG0 = 4, EMIT_SEG1 = 8 };

// rays and samples of a thread's steps (conn: MIS rays of unidirectional paths, connections of
// bidirectional ones)
struct LogicCounts {
  unsigned rays = 0, ext = 0, shadow = 0, conn = 0, trav = 0, samples = 0, prim = 0;
};

// The pathtracer prologue and createRay (udpt.cl:158-189, 213-238): the seed of pixel (px, py) of
// a pass and the direction of its camera ray. Double precision runs at a small fraction of the
// other rates: the step of the batch engine that starts paths between its shading with a
// division for each coordinate made eight mixed jobs take 77.4 ms, now 76.4.
__device__ __forceinline__ f4 camera_direction(const PassParams& pp, int px, int py, uint32_t rand, uint32_t& seed) {
  seed = (uint32_t)((py + 1) * pp.width + (px + 1));
  seed = rand * seed;
  seed = ym::wang_hash(seed);
  if (seed == 0) seed = ym::wang_hash(seed);
  const float r1 = draw(seed);
  const float r2 = draw(seed);
  const float fx = ym::add((float)px, r1), fy = ym::add((float)py, r2);
  f4 dir;
  dir.x = (float)(pp.aspect * (ym::divided(2.0 * (double)fx, pp.w, pp.inv_w) - 1.0));
  dir.y = (float)(ym::divided(2.0 * (double)fy, pp.h, pp.inv_h) - 1.0);
  dir.z = -pp.cam.view_plane_dist;
  dir.w = 0.0f;
  f4 d;
  d.x = ym::dot(ld4(pp.cam.r1), dir);
  d.y = ym::dot(ld4(pp.cam.r2), dir);
  d.z = ym::dot(ld4(pp.cam.r3), dir);
  d.w = ym::dot(ld4(pp.cam.r4), dir);
  return ym::normalize(d);
}

// The power function and the normalisation, called. A shading step holds six of one and ten of
// the other; inlined they were a fifth of its code, and with two or three warps a scheduler in
// different places of it the kernels wait for instructions (5.0-5.2 stalls per issue in the
// tail of a 256x256 frame of the Cornell box, 2.9 now): a 256x256 frame of the Cornell box 0.62 -> 0.55 ms, four 512x512 passes 3.87 -> 3.53, the
// 1024x1024 glass sphere 5.35 -> 5.15, two MIS passes 4.17 -> 4.05. (Fresnel, refraction, the
// Oren-Nayar term, the light loops, the surface point, sine, root or reciprocal called as well:
// slower or alike.)
static __device__ __noinline__ float power(float x, float y) { return ym::pow(x, y); }
static __device__ __noinline__ f4 unit(f4 v) { return ym::normalize(v); }

struct Vtx {
  f4 hp;      // hit point, w = 1
  f4 n;       // shading normal, w = 0
  int mat;
};

// The device copies of a scene's quad lights carry, in fields the kernels do not read otherwise,
// values that depend on the lights alone, computed once on the host by the same operations
// (prepare_lights): in the padding the lengths of a light's edges and of its emission, in kd
// the power-proportional choice among the lights: the sum of the weights
// (ke.r + ke.g + ke.b) * area, this light's weight, its share, and the area density of a point
// sampled on it.
inline void prepare_lights(yc_quad_light* L, int n) {
  auto f = [](const yc_float4& v) { return ym::mk(v.x, v.y, v.z, v.w); };
  float total = 0.0f;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    L[i].pad[0] = ym::length(f(L[i].edge_l));
    L[i].pad[1] = ym::length(f(L[i].edge_w));
    L[i].pad[2] = ym::length(f(L[i].ke));
    L[i].kd.y = ym::mul(ym::add(ym::add(L[i].ke.x, L[i].ke.y), L[i].ke.z), ym::mul(L[i].pad[0], L[i].pad[1]));
    total = ym::add(total, L[i].kd.y);
  }
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    L[i].kd.x = total;
    L[i].kd.z = ym::div(L[i].kd.y, total);
    L[i].kd.w = ym::div(L[i].kd.z, ym::mul(L[i].pad[0], L[i].pad[1]));
  }
}
__device__ __forceinline__ float light_len_l(const yc_quad_light& L) { return L.pad[0]; }
__device__ __forceinline__ float light_len_w(const yc_quad_light& L) { return L.pad[1]; }
__device__ __forceinline__ float light_len_ke(const yc_quad_light& L) { return L.pad[2]; }
__device__ __forceinline__ float light_area(const yc_quad_light& L) { return ym::mul(light_len_l(L), light_len_w(L)); }
__device__ __forceinline__ float light_total(const yc_quad_light& L) { return L.kd.x; }
__device__ __forceinline__ float light_weight(const yc_quad_light& L) { return L.kd.y; }
__device__ __forceinline__ float light_share(const yc_quad_light& L) { return L.kd.z; }
__device__ __forceinline__ float light_point_pdf(const yc_quad_light& L) { return L.kd.w; }

// the analytic quad-light loop of traceRay (udpt.cl:244-276); updates len and the hit light
// (the loops over lights are not unrolled, for the same reason: eight mixed jobs 76.5 -> 75.6 ms)
__device__ __forceinline__ void light_test(const DevScene& sc, f4 o, f4 d, float& len, int& light) {
#pragma unroll 1
  for (int i = 0; i < sc.n_lights; ++i) {
    const yc_quad_light& L = sc.lights[i];
    const f4 nrm = ld4(L.normal);
    const float DdotN = ym::dot(d, nrm);
    if (ym::fabs(DdotN) > __uint_as_float(LIGHT_DDOTN_BITS)) {
      const f4 pos = ld4(L.pos);
      const float t = ym::div(ym::dot(nrm, pos - o), DdotN);
      if (t > 0.0f && t < len) {
        f4 temp = o + d * t;
        temp = temp - pos;
        const f4 el = ld4(L.edge_l), ew = ld4(L.edge_w);
        float p1 = ym::dot(temp, el);
        float p2 = ym::dot(temp, ew);
        const float la = light_len_l(L), lb = light_len_w(L);
        p1 = ym::div(p1, la);
        p2 = ym::div(p2, lb);
        if ((p1 >= 0.0f && p2 >= 0.0f) && (p1 <= la && p2 <= lb)) {
          len = t;
          light = i;
        }
      }
    }
  }
}

__device__ __forceinline__ void frame(f4 Nz, f4& Nx, f4& Ny) {
  if (ym::fabs(Nz.y) > ym::fabs(Nz.z)) Nx = ym::mk(Nz.y, -Nz.x, 0.0f, 0.0f);
  else Nx = ym::mk(Nz.z, 0.0f, -Nz.x, 0.0f);
  Nx = unit(Nx);
  Ny = unit(ym::cross(Nz, Nx));
}

// reflect, udpt.cl:949-961
__device__ __forceinline__ f4 reflect(f4 w_i, f4 n) {
  if (ym::dot(w_i, n) < 0.0f) n = n * -1.0f;
  const f4 r = ym::mul(2.0f, ym::dot(w_i, n)) * n - w_i;
  return unit(r);
}

// refract, udpt.cl:963-990
__device__ __forceinline__ f4 refract(f4 w_i, f4 n, float ior) {
  float n1, n2;
  if (ym::dot(w_i, n) < 0.0f) { n1 = ior; n2 = 1.0f; n = n * -1.0f; }
  else { n1 = 1.0f; n2 = ior; }
  const f4 perp = ym::div(n1, n2) * (ym::dot(w_i, n) * n - w_i);
  const float lp = ym::length(perp);
  const f4 par = ym::sqrt(ym::sub(1.0f, ym::mul(lp, lp))) * (-n);
  return unit(perp + par);
}

// evalFresnelReflectance, udpt.cl:992-1031
__device__ __forceinline__ float fresnel(f4 w_i, f4 n, const yc_material& m, float& ior_factor) {
  float n1, n2;
  if (ym::dot(w_i, n) < 0.0f) { n1 = m.n; n2 = 1.0f; n = n * -1.0f; }
  else { n1 = 1.0f; n2 = m.n; }
  const float cI = ym::dot(w_i, n);
  const float sI = ym::sqrt(ym::sub(1.0f, ym::mul(cI, cI)));
  const float sT = ym::div(ym::mul(n1, sI), n2);
  const float cT = ym::sqrt(ym::sub(1.0f, ym::mul(sT, sT)));
  if (sT >= 1.0f && n1 > n2) return 1.0f;
  const float r0 = ym::div(ym::add(ym::add(m.ks.x, m.ks.y), m.ks.z), 3.0f);
  ior_factor = ym::div(ym::mul(n2, n2), ym::mul(n1, n1));
  const float c = (n1 > n2) ? cI : cT;
  return ym::add(r0, ym::mul(ym::sub(1.0f, r0), ym::sub(1.0f, power(c, 5.0f))));
}

// normal-to-world rows (Nx.k, Ny.k, Nz.k, p.k) applied to (x, y, z, 0), then normalised
__device__ __forceinline__ f4 to_world(f4 Nx, f4 Ny, f4 Nz, f4 p, f4 d) {
  f4 o;
  o.x = ym::dot(ym::mk(Nx.x, Ny.x, Nz.x, p.x), d);
  o.y = ym::dot(ym::mk(Nx.y, Ny.y, Nz.y, p.y), d);
  o.z = ym::dot(ym::mk(Nx.z, Ny.z, Nz.z, p.z), d);
  o.w = 0.0f;
  return unit(o);
}

// A direction around the axis Nz (phongSampleHemisphere, udpt.cl:700-771, and
// cosineWeightedHemisphere, udpt.cl:843-910, differ in the axis, the polar angle and the
// density): one code for both, so that lanes with either lobe run it together. `lobe`: the
// modified Phong lobe of exponent pe around Nz; otherwise the cosine lobe, Nz = v.n.
__device__ __forceinline__ f4 sample_around(const Vtx& v, f4 Nz, bool lobe, int pe, uint32_t& seed, float& pdf) {
  f4 Nx, Ny;
  frame(Nz, Nx, Ny);
  const float r1 = draw(seed);
  const float r2 = draw(seed);
  const float phi = ym::mul(ym::mul(2.0f, PI_F), r2);
  float st, ct;
  if (lobe) {
    ct = power(r1, ym::rcp((float)(pe + 1)));
    st = ym::sqrt(ym::sub(1.0f, power(r1, ym::div(2.0f, (float)(pe + 1)))));
  } else {
    st = ym::sqrt(r1);
    ct = ym::sqrt(ym::sub(1.0f, r1));
  }
  float sn, cs;
  ym::sincos(phi, sn, cs);
  const f4 dir = to_world(Nx, Ny, Nz, v.hp, ym::mk(ym::mul(st, cs), ym::mul(st, sn), ct, 0.0f));
  if (!lobe) pdf = ym::mul(ct, INV_PI_F);
  else if (ym::dot(dir, v.n) < 0.0f) pdf = 0.0f;
  else pdf = (float)((double)(pe + 1) * 0.5 * (double)INV_PI_F * (double)power(ct, (float)pe));
  return dir;
}
__device__ __forceinline__ f4 sample_cosine(const Vtx& v, uint32_t& seed, float& pdf) {
  return sample_around(v, v.n, false, 0, seed, pdf);
}
// the diffuse or the glossy lobe of m seen from w_i (direction and pdf; origin = hp + dir * EPS)
__device__ __forceinline__ f4 sample_lobe(const Vtx& v, const yc_material& m, bool glossy, f4 w_i, uint32_t& seed,
                                          float& pdf) {
  const f4 Nz = glossy ? unit(reflect(w_i, v.n)) : v.n;
  return sample_around(v, Nz, glossy, (int)ym::add(m.px, m.py), seed, pdf);
}

// calcPhongPDF, udpt.cl:1033-1045
__device__ __forceinline__ float phong_pdf(f4 w_i, f4 w_o, const Vtx& v, const yc_material& m) {
  f4 rd = ym::mul(2.0f, ym::dot(w_o, v.n)) * v.n - w_o;
  rd = unit(rd);
  const float ct = ym::fmax(0.0f, ym::cos(ym::dot(rd, w_i)));
  const float pe = ym::add(m.px, m.py);
  return (float)((double)ym::add(pe, 1.0f) * 0.5 * (double)INV_PI_F * (double)power(ct, pe));
}
// calcCosPDF, udpt.cl:1047-1050
__device__ __forceinline__ float cos_pdf(f4 w_i, f4 n) { return ym::mul(ym::fmax(ym::dot(w_i, n), 0.0f), INV_PI_F); }

// sampleGlossyPdf, udpt.cl:1062-1119
__device__ __forceinline__ bool sample_glossy(const yc_material& m, uint32_t& seed, float& prob) {
  const float r = draw(seed);
  const f4 ks = ld4(m.ks), kd = ld4(m.kd);
  if (ym::length3(ks) == 0.0f) { prob = 1.0f; return false; }
  if (ym::length3(kd) == 0.0f || ym::add(ym::add(kd.x, kd.y), kd.z) == 0.0f) { prob = 1.0f; return true; }
  const f4 sum = ks + kd;
  const float mx = ym::max(sum.x, ym::max(sum.y, sum.z));
  float pd, ps;
  if (mx == sum.x) { pd = kd.x; ps = ks.x; }
  else if (mx == sum.y) { pd = kd.y; ps = ks.y; }
  else { pd = kd.z; ps = ks.z; }
  if (r < pd) { prob = pd; return false; }
  if (r < ym::add(pd, ps) && r >= pd) { prob = ps; return true; }
  prob = 0.0f;
  return false;
}

// toShadingSpace + trig helpers, udpt-primitives.cl:1147-1210
__device__ __forceinline__ f4 to_shading(f4 w, const Vtx& v) {
  f4 Nx, Ny;
  frame(v.n, Nx, Ny);
  const f4 Nz = v.n;
  const f4 r1 = ym::mk(Nx.x, Nx.y, Nx.z, ym::dot(v.hp, Nx));
  const f4 r2 = ym::mk(Ny.x, Ny.y, Ny.z, ym::dot(v.hp, Ny));
  const f4 r3 = ym::mk(Nz.x, Nz.y, Nz.z, ym::dot(v.hp, Nz));
  const f4 r4 = ym::mk(0.0f, 0.0f, 0.0f, 1.0f);
  return ym::mk(ym::dot(r1, w), ym::dot(r2, w), ym::dot(r3, w), ym::dot(r4, w));
}
__device__ __forceinline__ float sin_theta(f4 w) { return ym::sqrt(ym::sub(1.0f, ym::mul(w.z, w.z))); }
__device__ __forceinline__ float cos_phi(f4 w) {
  const float st = sin_theta(w);
  if (st <= EPS_F && st >= -EPS_F) return 0.0f;
  return ym::clamp(ym::div(w.x, st), -1.0f, 1.0f);
}
__device__ __forceinline__ float sin_phi(f4 w) {
  const float st = sin_theta(w);
  if (st <= EPS_F && st >= -EPS_F) return 0.0f;
  return ym::clamp(ym::div(w.y, st), -1.0f, 1.0f);
}
// OrenNayarBRDF, udpt-primitives.cl:696-725 (alpha_x holds sigma^2). A and B (:722-723) depend on
// the material alone and are computed in double precision; oren_nayar_ab (host and
// device) is that computation, done once per material at upload (DevScene::on_ab), so a
// shading step runs no double-precision division.
__host__ __device__ inline float2 oren_nayar_ab(float alpha_x) {
  const double s2 = (double)alpha_x;
  float2 ab;
  ab.x = (float)(1 - (s2 / (2 * (s2 + 0.33))));
  ab.y = (float)(0.45 * s2 / (s2 + 0.09));
  return ab;
}
__device__ __forceinline__ f4 oren_nayar(f4 w_i, f4 w_o, const Vtx& v, const yc_material& m, float2 ab) {
  w_i = to_shading(w_i, v);
  w_o = to_shading(w_o, v);
  float costerm = 0.0f;
  if (sin_theta(w_i) >= EPS_F && sin_theta(w_o) >= EPS_F)
    costerm = ym::fmax(0.0f, ym::add(ym::mul(cos_phi(w_i), cos_phi(w_o)), ym::mul(sin_phi(w_i), sin_phi(w_o))));
  float sa, tb;
  if (ym::fabs(w_i.z) < ym::fabs(w_o.z)) { sa = sin_theta(w_i); tb = ym::div(sin_theta(w_o), ym::fabs(w_o.z)); }
  else { sa = sin_theta(w_o); tb = ym::div(sin_theta(w_i), ym::fabs(w_i.z)); }
  return (ld4(m.kd) * INV_PI_F) * ym::add(ab.x, ym::mul(ab.y, ym::mul(ym::mul(costerm, sa), tb)));
}

// evaluateBRDF, udpt.cl:611-630 (Oren-Nayar for a probability-1 diffuse lobe when
// brdf_model = 1, udpt-primitives.cl:673-686; on_ab: the scene's per-material A and B)
__device__ __forceinline__ f4 brdf(f4 w_i, f4 w_o, const Vtx& v, const yc_material& m, bool glossy, float rr_prob,
                                   int brdf_model, const float2* on_ab) {
  if (!glossy) {
    if (brdf_model == 1 && rr_prob == 1.0f) return oren_nayar(w_i, w_o, v, m, on_ab[v.mat]);
    return (ld4(m.kd) * INV_PI_F) / rr_prob;
  }
  const f4 refl = unit(reflect(w_i, v.n));
  const float ca = power(ym::fmax(ym::dot(w_o, refl), 0.0f), ym::add(m.px, m.py));
  const int pe = (int)ym::add(m.px, m.py);
  return ((((ld4(m.ks) * ca) * (float)(pe + 2)) * INV_PI_F) * 0.5f) / rr_prob;
}

// sampleLights, udpt.cl:632-698; -1 when no light is picked
__device__ __forceinline__ int sample_lights(const DevScene& sc, const Vtx& v, uint32_t& seed, float& light_pdf,
                                             f4& w_i) {
  // The reference keeps each light's sample and weight in arrays; here the weights are
  // summed in a first sweep and the chosen light's sample is drawn again in a second
  // sweep that replays the same xorshift stream, so nothing is spilled to local memory
  // and every value is computed by the same operations in the same order.
  const int n = sc.n_lights;
  const uint32_t seed0 = seed;
  float sum = 0.0f;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const yc_quad_light& L = sc.lights[i];
    const float r1 = draw(seed);
    const float r2 = draw(seed);
    f4 t = ((ld4(L.pos) + r1 * ld4(L.edge_l)) + r2 * ld4(L.edge_w)) - v.hp;
    const float distance = ym::dot(t, t);
    const f4 ti = t;
    t = unit(t);
    const f4 ln = ld4(L.normal);
    const float cf = ym::mul(ym::max(ym::dot(t, v.n), 0.0f), ym::max(ym::dot(-t, ln), 0.0f));
    if (cf <= 0.0f) continue;
    const float area = light_area(L);
    if (n == 1) {
      w_i = ti;
      light_pdf = ym::rcp(area);
      light_pdf = ym::mul(light_pdf, ym::div(distance, ym::fmax(ym::dot(-t, ln), 0.0f)));
      return i;
    }
    sum = ym::add(sum, ym::div(ym::mul(ym::mul(light_len_ke(L), cf), area), distance));
  }
  if (sum == 0.0f) return -1;
  const float r1 = draw(seed);
  float cum = 0.0f;
  uint32_t replay = seed0;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const yc_quad_light& L = sc.lights[i];
    const float q1 = draw(replay);
    const float q2 = draw(replay);
    f4 t = ((ld4(L.pos) + q1 * ld4(L.edge_l)) + q2 * ld4(L.edge_w)) - v.hp;
    const float distance = ym::dot(t, t);
    const f4 ti = t;
    t = unit(t);
    const f4 ln = ld4(L.normal);
    const float cf = ym::mul(ym::max(ym::dot(t, v.n), 0.0f), ym::max(ym::dot(-t, ln), 0.0f));
    const float area = light_area(L);
    const float weight = cf <= 0.0f ? 0.0f : ym::div(ym::mul(ym::mul(light_len_ke(L), cf), area), distance);
    const float wgt = ym::div(weight, sum);
    if (r1 >= cum && r1 < ym::add(cum, wgt)) {
      w_i = ti;
      light_pdf = ym::div(wgt, area);
      light_pdf = ym::mul(light_pdf, ym::div(ym::dot(w_i, w_i), ym::fmax(ym::dot(-unit(w_i), ln), 0.0f)));
      return i;
    }
    cum = ym::add(cum, wgt);
  }
  return -1;
}

// ---- the BDPT variants (kernels/legacy/bdpt.cl) ----
// evaluateBRDF, bdpt.cl:718-737: reflection vector without the normal flip
__device__ __forceinline__ f4 brdf_b(f4 w_i, f4 w_o, f4 n, const yc_material& m, bool glossy, float rr_prob) {
  f4 refl = ym::mul(2.0f, ym::dot(w_i, n)) * n - w_i;
  refl = unit(refl);
  if (!glossy) return (ld4(m.kd) * INV_PI_F) / rr_prob;
  const float ca = power(ym::fmax(ym::dot(w_o, refl), 0.0f), ym::add(m.px, m.py));
  const int pe = (int)ym::add(m.px, m.py);
  return ((((ld4(m.ks) * ca) * (float)(pe + 2)) * INV_PI_F) * 0.5f) / rr_prob;
}

// the diffuse or the glossy lobe (phongSampleHemisphere, bdpt.cl:807-870: lobe axis
// without the normal flip)
__device__ __forceinline__ f4 sample_lobe_b(const Vtx& v, const yc_material& m, bool glossy, f4 w_i, uint32_t& seed,
                                            float& pdf) {
  const f4 Nz = glossy ? unit(ym::mul(2.0f, ym::dot(w_i, v.n)) * v.n - w_i) : v.n;
  return sample_around(v, Nz, glossy, (int)ym::add(m.px, m.py), seed, pdf);
}

// sampleGlossyPdf, bdpt.cl:1048-1105: probabilities raised by (1 - max)/2, no absorption
__device__ __forceinline__ bool sample_glossy_b(const yc_material& m, uint32_t& seed, float& prob) {
  const float r = draw(seed);
  const f4 ks = ld4(m.ks), kd = ld4(m.kd);
  if (ym::length3(ks) == 0.0f) { prob = 1.0f; return false; }
  if (ym::length3(kd) == 0.0f || ym::add(ym::add(kd.x, kd.y), kd.z) == 0.0f) { prob = 1.0f; return true; }
  const f4 sum = ks + kd;
  const float mx = ym::max(sum.x, ym::max(sum.y, sum.z));
  float pd, ps;
  if (mx == sum.x) { pd = kd.x; ps = ks.x; }
  else if (mx == sum.y) { pd = kd.y; ps = ks.y; }
  else { pd = kd.z; ps = ks.z; }
  if (mx < 1.0f) {
    const float half = ym::div(ym::sub(1.0f, mx), 2.0f);
    pd = ym::add(pd, half);
    ps = ym::add(ps, half);
  }
  if (r < pd) { prob = pd; return false; }
  prob = ps;
  return true;
}

// getYluminance, udpt.cl:1121-1124
__device__ __forceinline__ float luminance(f4 c) {
  return ym::add(ym::add(ym::mul(0.212671f, c.x), ym::mul(0.715160f, c.y)), ym::mul(0.072169f, c.z));
}

// vertex of a triangle hit: hit point and interpolated normal (udpt.cl:377-383)
__device__ __forceinline__ Vtx tri_vertex(const DevScene& sc, f4 o, f4 d, float t, float u, float v, int tri) {
  Vtx x;
  x.hp = o + d * t;
  const float4* s = sc.shade + 4 * (size_t)tri;
  const f4 N1 = f4of(__ldg(s + 0)), N2 = f4of(__ldg(s + 1)), N3 = f4of(__ldg(s + 2));
  const float w = ym::sub(ym::sub(1.0f, u), v);
  x.n = unit((N1 * w + N2 * u) + N3 * v);
  x.mat = __float_as_int(__ldg(s + 3).x);
  return x;
}

}  // namespace yc
