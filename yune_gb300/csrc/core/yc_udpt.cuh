// yc_udpt.cuh -- the unidirectional path's per-path device logic (kernels/legacy/udpt.cl),
// shared by the per-pass kernels (udpt.cu) and the batch engine (engine.cu).
#pragma once

#include "yc_internal.h"
#include "yc_shade.cuh"

namespace yc {

enum : int {
  S_PRIMARY = 0,     // waiting for the closest hit of the camera ray
  S_NEE_SHADOW = 1,  // waiting for the shadow ray of evaluateDirectLighting
  S_NEE_MIS = 2,     // waiting for the MIS BRDF ray (any-hit up to the sampled light)
  S_EXT = 3,         // waiting for the closest hit of the GI extension ray
  // transient phases
  P_NEE_BEGIN = 8,
  P_NEE_DELIVER = 9,
  P_GI_SAMPLE = 10,
  P_FINISH = 11
};
enum : int {
  F_TARGET_INDIRECT = 1,  // NEE result goes to indirect += thr * DL (udpt.cl:527) else direct = DL
  F_NEE_GLOSSY = 2,       // sample_glossy of the NEE (udpt.cl:559)
  F_SPEC = 4,             // the pending extension ray left a specular vertex
  F_OCCLUDED = 8          // the NEE shadow ray was blocked
};

__device__ __forceinline__ int pack_misc(int state, int flags, int j, int k) {
  return state | (flags << 4) | ((j + 1) << 12) | ((k + 1) << 20);
}

constexpr int LOGIC_TB = 256;

struct LogicCounts {
  unsigned rays = 0, ext = 0, shadow = 0, mis = 0, trav = 0, samples = 0, prim = 0;
};

// ---- raygen: pathtracer prologue + createRay (udpt.cl:158-189, 213-238) ----
// seed of pixel (px, py) for pass seed `rand`, the camera ray, and the closest light
// along it (the light loop of traceRay runs before the BVH, udpt.cl:244-276)
__device__ __forceinline__ void camera_ray(const PassParams& pp, int px, int py, uint32_t rand, uint32_t& seed, f4& o, f4& d,
                           float& len, int& k) {
  const int W = pp.width, H = pp.height;
  seed = (uint32_t)((py + 1) * W + (px + 1));
  seed = rand * seed;
  seed = ym::wang_hash(seed);
  if (seed == 0) seed = ym::wang_hash(seed);
  const float r1 = draw(seed);
  const float r2 = draw(seed);
  const float fx = ym::add((float)px, r1), fy = ym::add((float)py, r2);
  const float aspect = pp.aspect;
  f4 dir;
  dir.x = (float)((double)aspect * ((2.0 * (double)fx / (double)W) - 1));
  dir.y = (float)((2.0 * (double)fy / (double)H) - 1);
  dir.z = -pp.cam.view_plane_dist;
  dir.w = 0.0f;
  d.x = ym::dot(ld4(pp.cam.r1), dir);
  d.y = ym::dot(ld4(pp.cam.r2), dir);
  d.z = ym::dot(ld4(pp.cam.r3), dir);
  d.w = ym::dot(ld4(pp.cam.r4), dir);
  d = ym::normalize(d);
  o = ym::mk(pp.cam.r1.w, pp.cam.r2.w, pp.cam.r3.w, pp.cam.r4.w);
  len = __int_as_float(0x7f800000);
  k = -1;
  light_test(pp.sc, o, d, len, k);
}

// Fields of the path record a step rewrote (stored back when the step emits a ray).
enum : unsigned {
  D_THR = 1, D_THR_NEXT = 2, D_DIRECT = 4, D_INDIRECT = 8, D_LS = 16, D_HP = 32, D_NRM = 64, D_WO = 128, D_WI = 256
};

// One step of path p: runs its state machine from the result of its last ray until it
// needs the next one. Returns 1 (closest-hit ray written to the path state), 2 (any-hit
// ray) or 0 (the path finished and its colour went into the accumulator). `mask`: the lanes
// of the warp that make the call together.
// The step loads only the record fields its entry state can read before writing them
// (a camera-ray result reads the ray and the hit; an extension result does not read the
// last vertex's shading frame, light sample or densities; a shadow or MIS result does not
// read the ray it traced) and stores only the fields it changed: the record is the same,
// with fewer bytes moved (pass starts write the misc word and the ray only).
__device__ __forceinline__ int logic_path(const PassParams& pp, int reset, const PathState& ps, int p, LogicCounts& cnt,
                                          unsigned mask) {
  const DevScene& sc = pp.sc;
  const f4 BG = ym::mk(0.4f, 0.4f, 0.4f, 1.0f);
  const f4 PINK = ym::mk(0.988f, 0.0588f, 0.7529f, 1.0f);
  const float INF = __int_as_float(0x7f800000);
  int emit = 0;
  int4 misc = ps.misc[p];
  uint32_t seed = (uint32_t)misc.x;
  const int pix = misc.y;
  int phase = misc.z & 15;
  int flags = (misc.z >> 4) & 0xff;
  int j = ((misc.z >> 12) & 0xff) - 1;
  int k = ((misc.z >> 20) & 0xff) - 1;
  int bounce = misc.w;
  const bool enter_cam = phase == S_PRIMARY, enter_ext = phase == S_EXT;
  const bool enter_nee = phase == S_NEE_SHADOW || phase == S_NEE_MIS;
  unsigned dirty = 0;
  const float4 Z4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  f4 thr = f4of(enter_cam ? Z4 : ps.thr[p]);
  f4 thr_next = f4of(enter_ext ? ps.thr_next[p] : Z4);
  f4 direct = f4of(enter_cam ? Z4 : ps.direct[p]), indirect = f4of(enter_cam ? Z4 : ps.indirect[p]);
  f4 ls = f4of(phase == S_NEE_MIS ? ps.ls[p] : Z4);
  const float4 hp4 = enter_nee ? ps.hp[p] : Z4, n4 = enter_nee ? ps.nrm[p] : Z4;
  const float4 wo4 = enter_nee ? ps.wo[p] : Z4, wi4 = enter_nee ? ps.wi[p] : Z4;
  Vtx V;
  V.hp = ym::mk(hp4.x, hp4.y, hp4.z, 1.0f);
  V.n = ym::mk(n4.x, n4.y, n4.z, 0.0f);
  V.mat = __float_as_int(wi4.w);
  float light_pdf = hp4.w, brdf_prob = n4.w, brdf_pdf = wo4.w;
  f4 wo = ym::mk(wo4.x, wo4.y, wo4.z, -0.0f);
  f4 w_i = ym::mk(wi4.x, wi4.y, wi4.z, 0.0f);
  const float4 ro4 = enter_nee ? Z4 : ps.ro[p], rd4 = enter_nee ? Z4 : ps.rd[p];
  f4 ro = ym::mk(ro4.x, ro4.y, ro4.z, 1.0f);
  f4 rd = ym::mk(rd4.x, rd4.y, rd4.z, rd4.w);
  float tmax = ro4.w;
  const float4 hit = ps.hit[p];
  f4 dl = ym::splat(0.0f);   // result of evaluateDirectLighting being delivered
  f4 color = ym::splat(0.0f);
  bool no_surface = false;   // the camera ray met no triangle: its colour is set

  // The result of a camera or extension ray: the vertex it met.
  if (enter_cam || enter_ext) {
    const int tri = __float_as_int(hit.w);
    const bool hit_tri = tri >= 0;
    Vtx NV = V;
    if (hit_tri) NV = tri_vertex(sc, ro, rd, hit.x, hit.y, hit.z, tri);
    if (enter_cam) {
      if (hit_tri) {
        thr = ym::mk(1.0f, 1.0f, 1.0f, 1.0f);
        direct = ym::mk(0.0f, 0.0f, 0.0f, 0.0f);
        indirect = direct;
        bounce = 0;
        flags = 0;
        dirty |= D_THR | D_DIRECT | D_INDIRECT | D_HP | D_NRM | D_WO | D_WI;
      } else {
        if (k >= 0) color = (ym::dot(rd, ld4(sc.lights[k].normal)) < 0.0f) ? ym::mk(1.0f, 1.0f, 1.0f, 1.0f)
                                                                           : ym::mk(0.1f, 0.1f, 0.1f, 1.0f);
        else color = BG;
        no_surface = true;
        phase = P_FINISH;
      }
    } else {   // rest of the GI iteration (udpt.cl:488-529)
      if (hit_tri) {
        indirect = indirect + thr * ld4(sc.mats[NV.mat].ke);
        thr = thr_next;
        dirty |= D_THR | D_INDIRECT | D_HP | D_NRM | D_WO | D_WI;   // new vertex
        if (bounce > pp.rr_threshold) {
          const float pr = ym::min(luminance(thr), 0.95f);
          const float r = draw(seed);
          if (r >= pr) phase = P_FINISH;
          else thr = thr * ym::div(1.0f, pr);
        }
        ++bounce;
      } else {
        if ((flags & F_SPEC) && k >= 0) indirect = indirect + thr * ld4(sc.lights[k].ke);
        phase = P_FINISH;
      }
    }
    if (phase != P_FINISH) {
      V = NV;
      wo = -rd;
      if (!sc.mats[V.mat].is_specular) {
        if (enter_ext) flags |= F_TARGET_INDIRECT;
        phase = P_NEE_BEGIN;
      } else {
        phase = P_GI_SAMPLE;
        if (enter_cam && !pp.gi_check) phase = P_FINISH;
      }
    }
  }
  // A ray to cast at the end of the iteration below: the state its result will be waited
  // for in, its direction and its length.
  int cast = 0;
  f4 dir = rd;
  float limit = INF;
  __syncwarp(mask);
  if (phase == P_NEE_BEGIN) {   // evaluateDirectLighting up to the shadow ray (udpt.cl:535-553)
    f4 wi_raw;
    j = sample_lights(sc, V, seed, light_pdf, wi_raw);
    if (j == -1 || light_pdf <= 0.0f) {
      dl = ld4(sc.mats[V.mat].ke);
      phase = P_NEE_DELIVER;
    } else {
      limit = ym::sub(ym::length(wi_raw), ym::mul(EPS_F, 1.5f));
      w_i = ym::normalize(wi_raw);
      flags &= ~(F_NEE_GLOSSY | F_OCCLUDED);
      dirty |= D_WI;
      dir = w_i;
      cast = S_NEE_SHADOW;
    }
  }
  // Each pass over the stages below takes a path one ray further: lobe choice, sampling,
  // BRDF and the light loop appear once in the code whichever ray they serve (the kernel
  // is bound by instruction fetch and by its lanes' different phases, so one copy that
  // the lanes of every phase share is worth the loop: a shadow result that goes on to
  // a MIS ray and a path that samples its next bounce run the same instructions). Most
  // paths leave after one pass; a MIS ray that misses the light takes a second one.
  // Measured against one copy per phase (a switch over the phases): 2.16 -> 1.69 ms of
  // shading per four 512x512 passes of the Cornell box, whose queue is not sorted, 1.11 ->
  // 0.97 ms per 1024x1024 pass of the glass sphere, whose queue is. The warp barriers keep
  // the compiler from sending lanes past the point where they meet again (without them
  // the same stages took 8% longer).
  for (;;) {
    __syncwarp(mask);
    if (phase == P_NEE_DELIVER) {
      if (flags & F_TARGET_INDIRECT) { indirect = indirect + thr * dl; dirty |= D_INDIRECT; }
      else { direct = dl; dirty |= D_DIRECT; }
      phase = pp.gi_check ? P_GI_SAMPLE : P_FINISH;
    }
    if (phase == P_GI_SAMPLE && bounce >= pp.max_depth) phase = P_FINISH;
    const bool waits = !cast && !emit;
    const bool shadow = waits && phase == S_NEE_SHADOW, mis_result = waits && phase == S_NEE_MIS;
    const bool gi = waits && phase == P_GI_SAMPLE;
    if (shadow || mis_result || gi) {
      const yc_material& m = sc.mats[V.mat];
      const bool spec = gi && m.is_specular != 0;
      if (shadow) {
        ls = ym::splat(0.0f);   // the light sample of this shadow ray (zero while occluded)
        dirty |= D_LS | D_NRM | D_WO;   // ls, brdf_prob, brdf_pdf
        if (hit.x != 0.0f) flags |= F_OCCLUDED;
        brdf_prob = 0.0f;
      }
      const bool visible = shadow ? !(flags & F_OCCLUDED) : hit.x == 0.0f;   // of a shadow or MIS result
      // lobe (sampleGlossyPdf): for the light sample and the MIS ray, or for the next bounce
      const bool draws = shadow ? visible || (pp.mis && pp.mis_lobe_fix) : gi && !spec;
      bool glossy = mis_result && (flags & F_NEE_GLOSSY);
      float prob = mis_result ? brdf_prob : 0.0f;
      if (draws) glossy = sample_glossy(m, seed, prob);
      if (shadow) brdf_prob = prob;
      // direction: the MIS ray's or the next bounce's (sampleFresnelIncidence, udpt.cl:912-947)
      const bool absorbed = draws && prob == 0.0f;
      const bool mis = shadow && pp.mis && !absorbed;
      const bool bounces = gi && !spec && !absorbed;
      f4 nd = dir;
      float pdf = absorbed ? 0.0f : 1.0f, ior = 1.0f;
      if (mis || bounces) nd = sample_lobe(V, m, glossy, wo, seed, pdf);
      if (spec) {
        bool mirrored = true;
        if (m.is_transmissive) {
          const float fr = fresnel(wo, V.n, m, ior);
          if (fr != 1.0f) mirrored = draw(seed) < fr;
        }
        if (mirrored) { nd = reflect(wo, V.n); ior = 1.0f; }
        else nd = refract(wo, V.n, m.n);
      }
      // BRDF: toward the light (light sample, MIS result) or along the next bounce
      const f4 to = gi ? nd : w_i;
      f4 f = ym::splat(0.0f);
      if (gi ? bounces && !(pdf <= 0.0f) : visible && !absorbed)
        f = brdf(to, wo, V, m, glossy, prob, pp.brdf_model, sc.on_ab);
      const float cosine = ym::fmax(ym::dot(to, V.n), 0.0f);
      if (gi) {   // one iteration of the GI loop up to its traceRay (udpt.cl:463-488)
        if (pdf <= 0.0f) {
          phase = P_FINISH;
        } else {
          thr_next = spec ? thr * ior : ((thr * f) * cosine) / pdf;
          dirty |= D_THR_NEXT;
          flags = spec ? (flags | F_SPEC) : (flags & ~F_SPEC);
          dir = nd;
          limit = INF;
          cast = S_EXT;
        }
      } else {    // evaluateDirectLighting after the shadow ray, or after the MIS ray (udpt.cl:553-608)
        const f4 em = ld4(m.ke);
        f4 x = (f * ld4(sc.lights[j].ke)) * cosine;
        const float mw = light_pdf;
        if (shadow) {
          if (visible && !absorbed) ls = x * ym::rcp(light_pdf);
          if (mis) {
            if (glossy) flags |= F_NEE_GLOSSY; else flags &= ~F_NEE_GLOSSY;
            brdf_pdf = glossy ? phong_pdf(w_i, wo, V, m) : cos_pdf(w_i, V.n);
            ls = ls * ym::div(ym::mul(mw, mw), ym::add(ym::mul(light_pdf, light_pdf), ym::mul(brdf_pdf, brdf_pdf)));
            brdf_pdf = pdf;
          }
          if (mis && !(pdf <= 0.0f)) {
            w_i = nd;
            dirty |= D_WI;
            dir = nd;
            limit = INF;
            cast = S_NEE_MIS;
          } else {
            dl = (visible && absorbed) ? em : ls + em;
            phase = P_NEE_DELIVER;
          }
        } else {
          dl = ls;
          if (visible) {
            const float w = ym::div(ym::mul(brdf_pdf, brdf_pdf),
                                    ym::add(ym::mul(light_pdf, light_pdf), ym::mul(brdf_pdf, brdf_pdf)));
            dl = ls + x * ym::div(w, brdf_pdf);
          }
          dl = dl + em;
          phase = P_NEE_DELIVER;
        }
      }
    }
    __syncwarp(mask);
    if (cast) {   // traceRay's light loop (udpt.cl:244-276); a ray that only the BVH can settle is emitted
      ro = V.hp + dir * EPS_F;
      rd = dir;
      float tl = limit;
      int lk = -1;
      light_test(sc, ro, rd, tl, lk);
      cnt.rays++;
      phase = cast;
      emit = cast == S_EXT ? 1 : 2;
      if (cast == S_NEE_SHADOW) {
        cnt.shadow++;
        tmax = limit;
        if (lk >= 0) {   // another light closes the segment: blocked without a BVH walk
          flags |= F_OCCLUDED;
          emit = 0;
        }
      } else if (cast == S_NEE_MIS) {   // only light j can satisfy the test
        cnt.mis++;
        tmax = tl;
        if (lk != j) {
          dl = ls + ld4(sc.mats[V.mat].ke);
          phase = P_NEE_DELIVER;
          emit = 0;
        }
      } else {
        cnt.ext++;
        tmax = tl;
        k = lk;
      }
      if (emit) cnt.trav++;
      cast = 0;
    }
    if (!__any_sync(mask, !emit && phase != P_FINISH)) break;
  }
  __syncwarp(mask);
  if (!emit) {   // the running mean of the pixel (udpt.cl:193-210)
    if (!no_surface) color = direct + indirect;
    if (ym::any_nan(color)) color = PINK;
    const float4 prev = pp.accum[pix];
    f4 c = color;
    if (reset == 1) {
      c.w = 1.0f;
    } else {
      const int np = (int)prev.w;
      c = c + f4of(prev) * (float)np;
      c = c / (float)(np + 1);
      c.w = (float)(np + 1);
    }
    pp.accum[pix] = make_float4(c.x, c.y, c.z, c.w);
    cnt.samples++;
  }
  if (emit) {
    ps.misc[p] = make_int4((int)seed, pix, pack_misc(phase, flags, j, k), bounce);
    if (dirty & D_THR) ps.thr[p] = make_float4(thr.x, thr.y, thr.z, thr.w);
    if (dirty & D_THR_NEXT) ps.thr_next[p] = make_float4(thr_next.x, thr_next.y, thr_next.z, thr_next.w);
    if (dirty & D_DIRECT) ps.direct[p] = make_float4(direct.x, direct.y, direct.z, direct.w);
    if (dirty & D_INDIRECT) ps.indirect[p] = make_float4(indirect.x, indirect.y, indirect.z, indirect.w);
    if (dirty & D_LS) ps.ls[p] = make_float4(ls.x, ls.y, ls.z, ls.w);
    if (dirty & D_HP) ps.hp[p] = make_float4(V.hp.x, V.hp.y, V.hp.z, light_pdf);
    if (dirty & D_NRM) ps.nrm[p] = make_float4(V.n.x, V.n.y, V.n.z, brdf_prob);
    if (dirty & D_WO) ps.wo[p] = make_float4(wo.x, wo.y, wo.z, brdf_pdf);
    if (dirty & D_WI) ps.wi[p] = make_float4(w_i.x, w_i.y, w_i.z, __int_as_float(V.mat));
    ps.ro[p] = make_float4(ro.x, ro.y, ro.z, tmax);
    ps.rd[p] = make_float4(rd.x, rd.y, rd.z, rd.w);
  }
  return emit;
}

}  // namespace yc
