// yc_udpt.cuh -- the unidirectional path's per-path device logic (kernels/legacy/udpt.cl),
// shared by the per-pass kernels (udpt.cu) and the batch engine (engine.cu).
#pragma once

#include "yc_internal.h"
#include "yc_shade.cuh"

namespace yc {

enum : int {
  S_PRIMARY = 0,     // waiting for the closest hit of the camera ray
  S_NEE_SHADOW = 1,  // waiting for the shadow ray of evaluateDirectLighting, to go on from there
  S_NEE_MIS = 2,     // waiting for the MIS BRDF ray (any-hit up to the sampled light), or only for
                     // the shadow ray in flight, nothing after it (F_LAST)
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
  F_OCCLUDED = 8,         // the NEE shadow ray was blocked
  F_WAIT = 16,            // a shadow ray is in flight beside the path's next ray (ls: the light sample if it is free)
  F_OCC_NAN = 32,         //   and if it is occluded the sample is NaN (0 times a weight without a value)
  F_LAST = 64             //   and it is the path's last ray
};
// the segments in flight of a path with this misc.z: shadow ray, MIS ray
__device__ __forceinline__ int segments_of(int state_flags) {
  const int state = state_flags & 15, flags = state_flags >> 4;
  return (state == S_NEE_SHADOW || (flags & F_WAIT) ? EMIT_SEG0 : 0) |
         (state == S_NEE_MIS && !(flags & F_LAST) ? EMIT_SEG1 : 0);
}

__device__ __forceinline__ int pack_misc(int state, int flags, int j, int k) {
  return state | (flags << 4) | ((j + 1) << 12) | ((k + 1) << 20);
}

constexpr int LOGIC_TB = 256;

// whether a vertex's shadow ray goes with the path's next ray (TOGETHER of logic_path)
inline bool rays_together(const PassParams& pp) { return pp.mis != 0 && pp.mis_lobe_fix != 0; }

// ---- raygen: pathtracer prologue + createRay (udpt.cl:158-189, 213-238) ----
// seed of pixel (px, py) for pass seed `rand`, the camera ray, and the closest light
// along it (the light loop of traceRay runs before the BVH, udpt.cl:244-276)
__device__ __forceinline__ void camera_ray(const PassParams& pp, int px, int py, uint32_t rand, uint32_t& seed, f4& o, f4& d,
                           float& len, int& k) {
  d = camera_direction(pp, px, py, rand, seed);
  o = ym::mk(pp.cam.r1.w, pp.cam.r2.w, pp.cam.r3.w, pp.cam.r4.w);
  len = __int_as_float(0x7f800000);
  k = -1;
  light_test(pp.sc, o, d, len, k);
}

// the first ray of pixel (px, py) in slot p
__device__ __forceinline__ void start_udpt(const PassParams& pp, const PathState& ps, int p, int px, int py, uint32_t rand) {
  uint32_t seed;
  f4 o, d;
  float len;
  int k;
  camera_ray(pp, px, py, rand, seed, o, d, len, k);
  ps.misc[p] = make_int4((int)seed, py * pp.width + px, pack_misc(S_PRIMARY, 0, -1, k), 0);
  ps.ro[p] = make_float4(o.x, o.y, o.z, len);
  ps.rd[p] = make_float4(d.x, d.y, d.z, d.w);
}

// ---- calls of several passes (MULTI) ----
// They run in one wavefront: a path that ends pass k of its pixel starts pass k + 1 in the next
// round (launch_raygen, or at once in the tail), so the rounds stay full and the call has one
// end with few paths, not one for each pass. Every pixel still adds its passes in order. Four
// 160x120 passes over 20K triangles 3.65 ms apart, 2.70 together, four of 800x600 over 60K 14.5 and 12.4.
__device__ __forceinline__ bool has_next_pass(const PassParams& pp, const PathState& ps, int p) {
  return ps.job[p].w + 1 < pp.n_pass;
}
// whether the path's pass starts the pixel's accumulator anew
__device__ __forceinline__ int pass_reset(const PassParams& pp, const PathState& ps, int p) {
  return ps.job[p].w > 0 ? 0 : pp.reset;
}

// Fields of the path record a step rewrote (stored back when the step emits a ray).
enum : unsigned { D_THR = 1, D_DIRECT = 4, D_INDIRECT = 8 };

// The queue entries of a warp's lanes (all 32 call it): paths with a closest-hit ray, paths that
// only wait for segments, and the segments; where each lane's entries went.
struct RaysOut {
  int closest, any;
};
__device__ __forceinline__ void append_rays(int emit, int p, int* out_closest, int* out_wait, int* q_any,
                                            RoundCounters* rc_out, RaysOut& at) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1;
  const bool closest = (emit & EMIT) == EMIT_CLOSEST, wait = (emit & EMIT) == EMIT_WAIT;
  const unsigned mc = __ballot_sync(0xffffffffu, closest), mw = __ballot_sync(0xffffffffu, wait);
  const unsigned m0 = __ballot_sync(0xffffffffu, (emit & EMIT_SEG0) != 0);
  const unsigned m1 = __ballot_sync(0xffffffffu, (emit & EMIT_SEG1) != 0);
  int bc = 0, bw = 0, ba = 0;
  if (lane == 0) {
    if (mc) bc = atomicAdd(&rc_out->n_closest, __popc(mc));
    if (mw) bw = atomicAdd(&rc_out->n_wait, __popc(mw));
    if (m0 | m1) ba = atomicAdd(&rc_out->n_any, __popc(m0) + __popc(m1));
  }
  at.closest = __shfl_sync(0xffffffffu, bc, 0) + __popc(mc & below);
  bw = __shfl_sync(0xffffffffu, bw, 0) + __popc(mw & below);
  at.any = __shfl_sync(0xffffffffu, ba, 0) + __popc(m0 & below) + __popc(m1 & below);
  if (closest) out_closest[at.closest] = p;
  if (wait) out_wait[bw] = p;
  int a = at.any;
  if (emit & EMIT_SEG0) q_any[a++] = 2 * p;
  if (emit & EMIT_SEG1) q_any[a] = 2 * p + 1;
}

// One step of path p: runs its state machine from the results of its last rays until it needs new
// ones. Returns what it sends (EMIT_*, the rays are in the path record), or 0 (the path finished
// and its colour went into the accumulator). `mask`: the lanes of the warp that make the call
// together.
// TOGETHER (rays_together): where the lobe is drawn whether the light is visible or not
// (mis_lobe_fix) no random number depends on the shadow ray's result, so the step goes on as if
// the ray were free and sends it with the path's next ray: the light sample waits in the record,
// and the next step takes it or leaves it, with the operations in the reference's order. A bounce
// is then one round for most paths instead of two or three, and the shading is as much work in
// fewer launches: four 512x512 passes of the Cornell box 4.77 -> 4.07 ms, a 256x256 frame of it
// 0.80 -> 0.70 ms, the 1024x1024 glass sphere 5.91 -> 5.60 ms. The MIS ray, which few paths
// need (most miss the light), stays alone: its share evaluated ahead as well, beside the
// extension ray, cost the shading kernel another pass of its loop for a few lanes (box 4.38 ms).
// A batch sends one ray at a time: its slots are always full, so a round less gains nothing.
// The step loads only the record fields its entry state can read before writing them and stores
// only the fields a later step reads.
template <bool TOGETHER>
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
  const bool enter_wait = TOGETHER && (flags & F_WAIT), enter_mis = phase == S_NEE_MIS && !(TOGETHER && (flags & F_LAST));
  const bool enter_nee = phase == S_NEE_SHADOW || enter_mis;
  unsigned dirty = 0;
  const float4 Z4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  f4 thr = f4of(enter_cam ? Z4 : ps.thr[p]);
  f4 thr_next = f4of(enter_ext ? ps.thr_next[p] : Z4);
  f4 direct = f4of(enter_cam ? Z4 : ps.direct[p]), indirect = f4of(enter_cam ? Z4 : ps.indirect[p]);
  f4 ls = f4of(enter_wait || enter_mis ? ps.ls[p] : Z4);
  const float4 hp4 = enter_nee || enter_wait ? ps.hp[p] : Z4, n4 = enter_nee ? ps.nrm[p] : Z4;
  const int occluded = (int)((unsigned)misc.z >> RECORD_BIT);   // bit 0: the shadow ray, bit 1: the MIS ray
  const float4 wo4 = enter_nee ? ps.wo[p] : Z4;
  Vtx V;
  V.hp = ym::mk(hp4.x, hp4.y, hp4.z, 1.0f);
  V.n = ym::mk(n4.x, n4.y, n4.z, 0.0f);
  V.mat = __float_as_int(hp4.w);
  f4 wo = ym::mk(wo4.x, wo4.y, wo4.z, -0.0f);
  const bool enter_hit = enter_cam || enter_ext;
  const float4 ro4 = enter_hit || enter_mis ? ps.ro[p] : Z4, hit = enter_hit ? ps.hit[p] : Z4;
  const float4 rd4 = enter_hit || enter_mis ? ps.rd[p] : enter_nee ? ps.wi[p] : Z4;
  float light_pdf = n4.w, brdf_prob = ro4.x, brdf_pdf = wo4.w;
  f4 w_i = ym::mk(rd4.x, rd4.y, rd4.z, 0.0f);   // (of a shadow or MIS ray)
  f4 ro = ym::mk(ro4.x, ro4.y, ro4.z, 1.0f);
  f4 rd = ym::mk(rd4.x, rd4.y, rd4.z, rd4.w);
  float tmax = ro4.w;
  f4 dl = ym::splat(0.0f);   // result of evaluateDirectLighting being delivered
  f4 color = ym::splat(0.0f);
  bool no_surface = false;   // the camera ray met no triangle: its colour is set

  // The light sample of the last vertex, now that its shadow ray is answered.
  if (enter_wait) {
    if (occluded & 1) ls = ym::splat(flags & F_OCC_NAN ? __int_as_float(0x7fffffff) : 0.0f);
    flags &= ~(F_WAIT | F_OCC_NAN);
    if (!enter_mis) {
      dl = ls + ld4(sc.mats[V.mat].ke);
      if (flags & F_TARGET_INDIRECT) { indirect = indirect + thr * dl; dirty |= D_INDIRECT; }
      else { direct = dl; dirty |= D_DIRECT; }
      if (!enter_ext) phase = P_FINISH;
    }
  }
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
        dirty |= D_THR | D_DIRECT | D_INDIRECT;
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
        dirty |= D_THR | D_INDIRECT;
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
      flags &= ~(F_NEE_GLOSSY | F_OCCLUDED | (TOGETHER ? F_OCC_NAN : 0));
      dir = w_i;
      cast = S_NEE_SHADOW;
    }
  }
  // Each pass over the stages below takes a path one ray further: lobe choice, sampling,
  // BRDF and the light loop appear once in the code whichever ray they serve (the kernel
  // is bound by instruction fetch and by its lanes' different phases, so one copy that
  // the lanes of every phase share is worth the loop: a shadow result that goes on to
  // a MIS ray and a path that samples its next bounce run the same instructions). Most
  // paths leave after one pass; a MIS ray that misses the light takes a second one, and a shadow
  // ray sent with the next ray one or two more.
  // Measured against one copy per phase (a switch over the phases): 2.16 -> 1.69 ms of
  // shading per four 512x512 passes of the Cornell box, whose queue is not sorted, 1.11 ->
  // 0.97 ms per 1024x1024 pass of the glass sphere, whose queue is. The warp barriers keep
  // the compiler from sending lanes past the point where they meet again (without them
  // the same stages took 8% longer).
  for (;;) {
    __syncwarp(mask);
    if (phase == P_NEE_DELIVER) {
      if (!TOGETHER || !(flags & F_WAIT)) {
        if (flags & F_TARGET_INDIRECT) { indirect = indirect + thr * dl; dirty |= D_INDIRECT; }
        else { direct = dl; dirty |= D_DIRECT; }
      }
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
        if (enter_nee && (occluded & 1)) flags |= F_OCCLUDED;   // (a ray still in flight counts as free)
        brdf_prob = 0.0f;
      }
      const bool visible = shadow ? !(flags & F_OCCLUDED) : !(occluded & 2);   // of a shadow or MIS result
      // lobe (sampleGlossyPdf): for the light sample and the MIS ray, or for the next bounce
      const bool draws = shadow ? TOGETHER || visible || (pp.mis && pp.mis_lobe_fix) : gi && !spec;
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
            const float weight =
                ym::div(ym::mul(mw, mw), ym::add(ym::mul(light_pdf, light_pdf), ym::mul(brdf_pdf, brdf_pdf)));
            ls = ls * weight;
            if (TOGETHER && !(weight < INF)) flags |= F_OCC_NAN;
            brdf_pdf = pdf;
          }
          if (mis && !(pdf <= 0.0f)) {
            w_i = nd;
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
    if (cast) {   // traceRay's light loop (udpt.cl:244-276); a ray that only the BVH can settle is sent
      ro = V.hp + dir * EPS_F;
      rd = dir;
      float tl = limit;
      int lk = -1;
      light_test(sc, ro, rd, tl, lk);
      cnt.rays++;
      phase = cast;
      tmax = tl;
      emit = EMIT_WAIT;
      if (cast == S_NEE_SHADOW) {
        cnt.shadow++;
        tmax = limit;
        if (lk >= 0) {   // another light closes the segment: blocked without a BVH walk
          flags |= F_OCCLUDED;
          emit = 0;
        } else if (TOGETHER) {
          ps.wi[p] = make_float4(dir.x, dir.y, dir.z, limit);
          flags |= F_WAIT;
          emit = 0;
          cnt.trav++;
        }
      } else if (cast == S_NEE_MIS) {   // only light j can satisfy the test
        cnt.conn++;
        if (lk != j) {
          dl = ls + ld4(sc.mats[V.mat].ke);
          phase = P_NEE_DELIVER;
          emit = 0;
        }
      } else {
        cnt.ext++;
        k = lk;
        emit = EMIT_CLOSEST;
      }
      if (emit) cnt.trav++;
      cast = 0;
    }
    if (TOGETHER && phase == P_FINISH && (flags & F_WAIT)) {   // the path ends, its last shadow ray is in flight
      phase = S_NEE_MIS;
      flags |= F_LAST;
      emit = EMIT_WAIT;
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
    if (dirty & D_DIRECT) ps.direct[p] = make_float4(direct.x, direct.y, direct.z, direct.w);
    if (dirty & D_INDIRECT) ps.indirect[p] = make_float4(indirect.x, indirect.y, indirect.z, indirect.w);
    const bool last = TOGETHER && (flags & F_LAST), wait = TOGETHER && (flags & F_WAIT);
    if (emit == EMIT_CLOSEST) {
      ps.thr_next[p] = make_float4(thr_next.x, thr_next.y, thr_next.z, thr_next.w);
      ps.ro[p] = make_float4(ro.x, ro.y, ro.z, tmax);
      ps.rd[p] = make_float4(rd.x, rd.y, rd.z, rd.w);
    } else if (!last) {   // evaluateDirectLighting goes on at this vertex
      ps.nrm[p] = make_float4(V.n.x, V.n.y, V.n.z, light_pdf);
      ps.wo[p] = make_float4(wo.x, wo.y, wo.z, brdf_pdf);
      (phase == S_NEE_MIS ? ps.rd[p] : ps.wi[p]) = make_float4(rd.x, rd.y, rd.z, tmax);
      if (phase == S_NEE_MIS) ps.ro[p].x = brdf_prob;
    }
    if (phase == S_NEE_MIS || wait) ps.ls[p] = make_float4(ls.x, ls.y, ls.z, ls.w);
    if (emit == EMIT_WAIT || wait) ps.hp[p] = make_float4(V.hp.x, V.hp.y, V.hp.z, __int_as_float(V.mat));
    emit |= segments_of(phase | (flags << 4));
  }
  return emit;
}

}  // namespace yc
