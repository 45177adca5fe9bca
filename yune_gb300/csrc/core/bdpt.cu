// bdpt.cu -- wavefront form of Yune's naive bidirectional path tracer
// (kernels/legacy/bdpt.cl:158-640), step (f) of the pipeline.
//
// Per sample the reference builds a light subpath (createLightPath, bdpt.cl:432-511),
// an eye subpath (createEyePath, bdpt.cl:513-560), then for every eye vertex adds its
// emission and next-event estimate and connects it to every light vertex j >= 1 with a
// shadow ray (shading, bdpt.cl:562-640). Here each path is a state machine like the
// unidirectional one (udpt.cu): the logic kernel advances it to its next subpath ray, or to
// all shadow rays of one eye vertex, the trace kernel settles both queues, and the subpath
// vertices live in HBM as one 64-byte record per vertex (two full 32-byte sectors: a
// connection reads two vertices of a path whose neighbours in the queue are unrelated),
// vertex k of path p at [(p * bounces + k) * 4 + field]:
//   field 0: hit point xyz, material index (int bits)
//   field 1: shading normal xyz
//   field 2: direction of the ray that reached the vertex xyz
//   field 3: contrib (the subpath throughput, float4)
// Random numbers are drawn in the reference order from the same per-pixel stream.
// One departure, shared with the CPU oracle: a camera ray that hits the light ends the
// eye path (the reference keeps extending it from a vertex with triangle_ID = -1 and
// reads scene_data[-1]; the pixel colour is fixed to white or grey either way).
#include <cuda_runtime.h>

#include "yc_bdpt.h"
#include "yc_shade.cuh"
#include "yc_tail.cuh"

namespace yc {

enum : int { BF_GLOSSY = 1 };
constexpr int CAST = 1;                         // a ray about to be sent: its state + CAST (0: none),
constexpr int TO_LIGHT = 8, TO_VERTEX = 9;      // or a segment's kind

struct BCount {
  int i, j, lp, ep;
};
__device__ __forceinline__ int pack_cnt(const BCount& c) { return c.i | (c.j << 6) | (c.lp << 12) | (c.ep << 18); }
__device__ __forceinline__ BCount unpack_cnt(int v) {
  return BCount{v & 63, (v >> 6) & 63, (v >> 12) & 63, (v >> 18) & 63};
}
__device__ __forceinline__ int pack_st(int state, int flags, int lj, int k) {
  return state | (flags << 4) | ((lj + 1) << 8) | ((k + 1) << 13);
}

struct VertexRef {
  float4* base;     // the path's first vertex
  __device__ __forceinline__ float4& at(int k, int f) const { return base[(size_t)k * 4 + f]; }
  __device__ __forceinline__ void store(int k, const Vtx& v, f4 dir, f4 contrib) const {
    at(k, 0) = make_float4(v.hp.x, v.hp.y, v.hp.z, __int_as_float(v.mat));
    at(k, 1) = make_float4(v.n.x, v.n.y, v.n.z, 0.0f);
    at(k, 2) = make_float4(dir.x, dir.y, dir.z, 0.0f);
    at(k, 3) = make_float4(contrib.x, contrib.y, contrib.z, contrib.w);
  }
  __device__ __forceinline__ Vtx vtx(int k) const {
    const float4 a = at(k, 0), b = at(k, 1);
    Vtx v;
    v.hp = ym::mk(a.x, a.y, a.z, 1.0f);
    v.n = ym::mk(b.x, b.y, b.z, 0.0f);
    v.mat = __float_as_int(a.w);
    return v;
  }
  __device__ __forceinline__ f4 dir(int k) const { const float4 d = at(k, 2); return ym::mk(d.x, d.y, d.z, 0.0f); }
  __device__ __forceinline__ f4 contrib(int k) const { return f4of(at(k, 3)); }
};

// ---- raygen: pixel prologue, eye ray, light vertex 0 and the first light ray ----
__global__ void __launch_bounds__(256) k_raygen_bdpt(PassParams pp, int n, int row, PathState ps,
                                                     BdptBuffers bb, int* q_closest, RoundCounters* rc, DevStats* st) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = gid < n;
  const int px = gid % row + pp.off_x, py = gid / row + pp.off_y;
  const int pix = py * pp.width + px;
  const int slot = pix;
  bool eye_first = false;
  if (active) {
    const DevScene& sc = pp.sc;
    uint32_t seed;
    const f4 d = camera_direction(pp, px, py, pp.rand_seed, seed);
    VertexRef ev{bb.ev + (size_t)slot * bb.bounces * 4};
    VertexRef lv{bb.lv + (size_t)slot * bb.bounces * 4};
    ev.at(0, 2) = make_float4(d.x, d.y, d.z, d.w);   // the camera ray, traced after the light subpath
    // light vertex 0 on light 0 (createLightPath, bdpt.cl:435-456)
    const yc_quad_light& L = sc.lights[0];
    seed = ym::xor_shift(seed);
    const float lr1 = ym::u01_inclusive(seed);
    const float lr2 = draw(seed);
    const f4 A = ld4(L.edge_l) * lr2;
    const f4 B = ld4(L.edge_w) * lr1;
    Vtx v0;
    v0.hp = (A + B) + ld4(L.pos);
    v0.n = ld4(L.normal);
    v0.mat = -1;
    const float fwd = ym::rcp(light_area(L));
    const f4 c0 = ld4(L.ke) / fwd;
    lv.at(0, 0) = make_float4(v0.hp.x, v0.hp.y, v0.hp.z, __int_as_float(-1));
    lv.at(0, 1) = make_float4(v0.n.x, v0.n.y, v0.n.z, v0.n.w);
    lv.at(0, 3) = make_float4(c0.x, c0.y, c0.z, c0.w);
    float pdf = 1.0f;
    const f4 ldir = sample_cosine(v0, seed, pdf);
    BCount cnt{1, 0, 1, 1};
    f4 o, rdir;
    int state;
    if (pdf <= 0.0f) {
      o = ym::mk(pp.cam.r1.w, pp.cam.r2.w, pp.cam.r3.w, pp.cam.r4.w);
      rdir = d;
      state = B_EYE0;
      cnt.i = 0;
      eye_first = true;
    } else {
      o = v0.hp + ldir * EPS_F;
      rdir = ldir;
      state = B_LIGHT;
    }
    float len = __int_as_float(0x7f800000);
    int k = -1;
    light_test(sc, o, rdir, len, k);
    ps.misc[slot] = make_int4((int)seed, pix, pack_st(state, 0, -1, k), pack_cnt(cnt));
    ps.ro[slot] = make_float4(o.x, o.y, o.z, len);
    ps.rd[slot] = make_float4(rdir.x, rdir.y, rdir.z, rdir.w);
    ps.direct[slot] = make_float4(1.0f, 0.0f, pdf, 0.0f);   // weight, ks, pending pdf, pending lobe prob
  }
  if (active) q_closest[gid] = slot;
  const unsigned eye = __ballot_sync(0xffffffffu, eye_first);   // (rare; counted with the light rays below)
  if (eye && (threadIdx.x & 31) == 0) {
    atomicAdd(&st->primary, (unsigned long long)__popc(eye));
    atomicAdd(&st->extension, 0ull - (unsigned long long)__popc(eye));
  }
  if (gid == 0) {
    rc->n_closest = n;
    atomicAdd(&st->rays, (unsigned long long)n);
    atomicAdd(&st->traversed, (unsigned long long)n);
    atomicAdd(&st->extension, (unsigned long long)n);
  }
}

void launch_raygen_bdpt(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, int* q_closest,
                        RoundCounters* rc, DevStats* st, cudaStream_t s) {
  const int n = tile_pixels(pp);
  if (n > 0) k_raygen_bdpt<<<(n + 255) / 256, 256, 0, s>>>(pp, n, tile_row(pp), ps, bb, q_closest, rc, st);
}

// ---- logic: advance each path to its next ray ----
// One step of path p: from the results of its last rays until it needs new ones. Returns what it
// sends (EMIT_*), or 0 (the path has ended). `mask`: the lanes of the warp that make the call together.
__device__ __forceinline__ int bdpt_step(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, int p,
                                         LogicCounts& lc, unsigned mask) {
  const DevScene& sc = pp.sc;
  const float INF = __int_as_float(0x7f800000);
  const int BOUNCES = bb.bounces;
  const int RR = 4;   // RR_THRESHOLD of bdpt.cl:4
  int emit = 0;
  FanOut out;   // the segments to send
  const VertexRef lv{bb.lv + (size_t)p * bb.bounces * 4};
  const VertexRef ev{bb.ev + (size_t)p * bb.bounces * 4};
  const int4 misc = ps.misc[p];
  uint32_t seed = (uint32_t)misc.x;
  const int pix = misc.y;
  int phase = misc.z & 15;
  int flags = (misc.z >> 4) & 15;
  int lj = ((misc.z >> 8) & 31) - 1;
  int k = ((misc.z >> 13) & 31) - 1;
  BCount cnt = unpack_cnt(misc.w);
  // While the subpaths are built (B_LIGHT, B_EYE0, B_EYE) the connection stage's
  // fields (colour, sub-sum, density of the light sample) are dead: Q_CONNECT initialises them.
  // They are loaded in the connection states only and stored once the stage has
  // started; the ray origin is read only where a hit point is built from it.
  const bool building = phase == B_LIGHT || phase == B_EYE0 || phase == B_EYE;
  bool conn_live = !building;
  f4 color = ym::splat(0.0f), sub = ym::splat(0.0f);
  float light_pdf = 0.0f;
  if (!building) {
    color = f4of(ps.thr[p]);
    sub = f4of(ps.thr_next[p]);
    light_pdf = ps.indirect[p].x;
  }
  float4 dv = ps.direct[p];
  float weight = dv.x, ks = dv.y, pend_pdf = dv.z, pend_prob = dv.w;
  f4 ro = ym::splat(0.0f), rd = ym::splat(0.0f);
  float tmax = 0.0f;
  if (building) {
    const float4 ro4 = ps.ro[p], rd4 = ps.rd[p];
    ro = ym::mk(ro4.x, ro4.y, ro4.z, 1.0f);
    rd = ym::mk(rd4.x, rd4.y, rd4.z, rd4.w);
    tmax = ro4.w;
  }
  const float4 hit = ps.hit[p];

  // ---- the result of the ray, or of the segments, the path waited for ----
  // A subpath ray's vertex takes the BRDF at the vertex the ray left; a free segment to a
  // light the BRDF at the eye vertex, a free one to a light vertex those at both ends, in
  // the order the reference connects them. One evaluation (lobe choice, BRDF) a pass for
  // each lane that has one left, so that one copy of the code serves them all.
  const bool light = phase == B_LIGHT, subpath = phase == B_LIGHT || phase == B_EYE;
  const int tri = __float_as_int(hit.w);
  const bool made = building && tri >= 0 && !(light && pend_pdf <= 0.0f);   // a vertex is made
  Vtx v, e;           // the vertex made; the eye vertex of the connection stage
  v.hp = v.n = e.hp = e.n = ym::splat(0.0f);
  v.mat = e.mat = 0;
  FanIn fan{0, 0};
  if (made) v = tri_vertex(sc, ro, rd, hit.x, hit.y, hit.z, tri);
  if (!building) {
    e = ev.vtx(cnt.i);
    fan.load(ps.job[p], misc);
    if (fan.vertex(0) == 0 && !(fan.free & 1u)) {   // the light sample is occluded: DL = emission
      const f4 em = ld4(sc.mats[e.mat].ke);
      color = color + (ev.contrib(cnt.i) * (em + (ym::splat(0.0f) + em))) * weight;
    }
  }
  f4 f0 = ym::splat(0.0f), pn = ym::splat(0.0f);
  bool left = made && subpath && !(light && cnt.i == 1);   // the BRDF where the subpath ray left
  bool far_end = false;                                    // of the first free segment
  for (;;) {
    const bool has = left || fan.free;
    if (!__any_sync(mask, has)) break;
    if (has) {
      Vtx at = e;
      f4 w_in = rd, w_out = rd, dir = ym::splat(0.0f);
      bool g = (flags & BF_GLOSSY) != 0;
      float prob = pend_prob;
      int j = 0;
      if (left) {
        const VertexRef& sv = light ? lv : ev;
        const f4 back = -sv.dir(cnt.i - 1);
        at = sv.vtx(cnt.i - 1);
        pn = at.n;
        if (light) w_in = back;
        else w_out = back;
      } else {
        const int sg = __ffs(fan.free) - 1;
        const float4 d4 = bb.seg[((size_t)p << bb.sg.shift) + sg];
        dir = ym::mk(d4.x, d4.y, d4.z, 0.0f);
        j = fan.vertex(sg);
        if (far_end) {
          at = lv.vtx(j);
          w_in = -lv.dir(j);
          w_out = -dir;
        } else {
          w_in = dir;
          w_out = -ev.dir(cnt.i);
        }
        g = sample_glossy_b(sc.mats[at.mat], seed, prob);
      }
      const f4 f = brdf_b(w_in, w_out, at.n, sc.mats[at.mat], g, prob);
      if (left) {
        f0 = f;
        left = false;
      } else if (j == 0) {   // the light sample, bdpt.cl:662-671 (MIS off, as shipped)
        const f4 em = ld4(sc.mats[e.mat].ke);
        f4 dl = em;
        if (prob != 0.0f) {
          f4 ls = (f * ld4(sc.lights[lj].ke)) * ym::fmax(ym::dot(dir, e.n), 0.0f);
          ls = ls * ym::div(1.0f, light_pdf);
          dl = ls + em;
        }
        color = color + (ev.contrib(cnt.i) * (em + dl)) * weight;
        fan.free &= fan.free - 1u;
      } else if (!far_end) {
        f0 = f;
        far_end = true;
      } else {               // a connection, bdpt.cl:616-634
        float dist = ym::length(at.hp - e.hp);
        dist = ym::mul(dist, dist);
        const float gf = ym::div(ym::mul(ym::max(ym::dot(dir, e.n), 0.0f), ym::max(ym::dot(-dir, at.n), 0.0f)), dist);
        f4 tlp = lv.contrib(j);
        tlp = tlp * ((gf * f0) * f);
        tlp = tlp * ev.contrib(cnt.i);
        sub = sub + tlp;
        far_end = false;
        fan.free &= fan.free - 1u;
      }
    }
  }
  if (building) {
    if (!made) {
      if (light) {
        phase = Q_EYE_START;
      } else if (phase == B_EYE) {
        phase = Q_CONNECT;
      } else {   // the camera ray met a light or nothing
        color = ym::mk(0.4f, 0.4f, 0.4f, 1.0f);
        if (k >= 0)
          color = (ym::dot(rd, ld4(sc.lights[k].normal)) < 0.0f) ? ym::mk(1.0f, 1.0f, 1.0f, 1.0f)
                                                                 : ym::mk(0.1f, 0.1f, 0.1f, 1.0f);
        phase = Q_FINISH;
      }
    } else {   // createLightPath (bdpt.cl:458-510), createEyePath (bdpt.cl:517-558)
      f4 contrib = ym::mk(1.0f, 1.0f, 1.0f, 1.0f);
      bool stop = false;
      const VertexRef& sv = light ? lv : ev;
      if (subpath) {
        if (light && cnt.i == 1) {
          const float c1 = ym::div(ym::max(0.0f, ym::dot(lv.vtx(0).n, rd)), pend_pdf);
          contrib = ym::splat(c1) * lv.contrib(0);
        } else {
          const float cosine = ym::dot(rd, pn);
          contrib = f0 * (light ? ym::fmax(0.0f, cosine) : ym::max(0.0f, cosine));
          contrib = contrib / pend_pdf;
          contrib = contrib * sv.contrib(cnt.i - 1);
        }
        if (cnt.i > RR) {
          const float r = draw(seed);
          const float pr = ym::min(luminance(contrib), 0.95f);
          if (r >= pr) stop = true;
          else contrib = contrib * ym::div(1.0f, pr);
        }
      } else {
        cnt.i = 0;
      }
      sv.store(cnt.i, v, rd, contrib);
      cnt.i += 1;
      if (light) cnt.lp = cnt.i;
      else cnt.ep = cnt.i;
      const bool full = cnt.i >= BOUNCES;
      phase = light ? (stop || full ? Q_EYE_START : Q_LIGHT_SAMPLE) : (stop || full ? Q_CONNECT : Q_EYE_SAMPLE);
    }
  } else {
    phase = Q_SEGMENTS;   // the vertex's light vertices not tried yet, if any
  }
  // ---- a subpath's next direction, from the vertex just made (bdpt.cl:473-484, 527-535) ----
  int cast = 0;           // the next ray: the state it will be waited for in + CAST, or a segment's kind
  f4 org = v.hp, dir = ym::splat(0.0f);
  float limit = INF;
  __syncwarp(mask);
  if (phase == Q_LIGHT_SAMPLE || phase == Q_EYE_SAMPLE) {
    const yc_material& m = sc.mats[v.mat];
    const bool on_light = phase == Q_LIGHT_SAMPLE;
    float prob = 0.0f, pdf = 1.0f;
    const bool g = sample_glossy_b(m, seed, prob);
    phase = on_light ? Q_EYE_START : Q_CONNECT;   // unless a direction is drawn
    if (prob != 0.0f) {
      dir = sample_lobe_b(v, m, g, -ym::mk(rd.x, rd.y, rd.z, 0.0f), seed, pdf);
      // (of the light subpath the reference traces before it tests the density, bdpt.cl:486)
      if (on_light || !(pdf <= 0.0f)) {
        flags = g ? (flags | BF_GLOSSY) : (flags & ~BF_GLOSSY);
        pend_pdf = pdf;
        pend_prob = prob;
        cast = on_light ? B_LIGHT + CAST : B_EYE + CAST;
      }
    }
  }
  if (phase == Q_EYE_START && !cast) {   // the camera ray (bdpt.cl:517-519)
    org = ym::mk(pp.cam.r1.w, pp.cam.r2.w, pp.cam.r3.w, pp.cam.r4.w);
    const float4 d = ev.at(0, 2);
    dir = ym::mk(d.x, d.y, d.z, d.w);
    cnt.i = 0;
    cast = B_EYE0 + CAST;
  }
  if (phase == Q_CONNECT && !cast) {   // shading starts (bdpt.cl:578-595)
    color = ym::mk(0.0f, 0.0f, 0.0f, 1.0f);
    weight = 1.0f;
    ks = 0.0f;
    cnt.i = cnt.j = 0;
    flags = 8;
    conn_live = true;
    phase = cnt.ep > 0 ? Q_VERTEX : Q_FINISH;
  }
  // ---- the connection stage until its next rays ----
  // The segments of an eye vertex, to the light sample and to every light vertex where both
  // ends face each other and no light is in between, are sent in one round (they depend on
  // no random number that a result draws): a path goes through as many rounds as it has
  // vertices, not segments. Each pass of the loop takes a lane past one light loop, which
  // serves every kind of ray. A round costs its launches and the chains of loads of its
  // last lanes, so fewer and larger ones pay in every kernel: a 1280x720 pass over 758K
  // triangles took 66 rounds and 15.3 ms with one segment a round, 24 rounds and 9.6 ms
  // with eight (trace 8.6 -> 5.2 ms, shading 3.6 -> 2.7, sorts 3.0 -> 1.7).
  for (;;) {
    __syncwarp(mask);
    if (phase == Q_VERTEX) {   // emission + next-event estimate at eye vertex i (bdpt.cl:591-597, 642-660)
      e = ev.vtx(cnt.i);
      const yc_material& m = sc.mats[e.mat];
      sub = ym::mk(0.0f, 0.0f, 0.0f, 1.0f);
      ks = ym::max(ym::max(m.ks.x, ym::max(m.ks.y, m.ks.z)), 0.1f);
      f4 wi_raw;
      lj = sample_lights(sc, e, seed, light_pdf, wi_raw);
      cnt.j = cnt.lp - 1;
      phase = Q_SEGMENTS;
      org = e.hp;
      if (lj == -1 || light_pdf <= 0.0f) {
        color = color + (ev.contrib(cnt.i) * (ld4(m.ke) + ld4(m.ke))) * weight;   // DL = emission
      } else {
        limit = ym::sub(ym::length(wi_raw), ym::mul(EPS_F, 1.5f));
        dir = ym::normalize(wi_raw);
        cast = TO_LIGHT;
      }
    }
    __syncwarp(mask);
    if (phase == Q_SEGMENTS && !cast) {   // the next connection j (bdpt.cl:598-615)
      org = e.hp;
      while (cnt.j > 0 && !cast && !out.full(bb)) {
        const float4 h4 = lv.at(cnt.j, 0), n4 = lv.at(cnt.j, 1);
        const f4 l_hp = ym::mk(h4.x, h4.y, h4.z, 1.0f), l_n = ym::mk(n4.x, n4.y, n4.z, 0.0f);
        dir = ym::normalize(l_hp - e.hp);
        if (ym::dot(dir, e.n) <= 0.0f || ym::dot(-dir, l_n) <= 0.0f) { cnt.j -= 1; continue; }
        limit = ym::length(l_hp - (e.hp + dir * EPS_F));
        cast = TO_VERTEX;
      }
      if (!cast) {
        if (out.n > 0) {
          phase = B_FAN;
          emit = 2;
        } else {   // every light vertex tried
          color = color + sub * ym::mul(weight, ym::sub(1.0f, ks));
          weight = ym::mul(weight, ks);
          cnt.i += 1;
          phase = cnt.i >= cnt.ep || weight == 0.0f ? Q_FINISH : Q_VERTEX;
        }
      }
    }
    __syncwarp(mask);
    if (cast) {   // traceRay's light loop (udpt.cl:244-276)
      const bool segment = cast >= TO_LIGHT;
      const f4 from = cast == B_EYE0 + CAST ? org : org + dir * EPS_F;
      float tl = limit;
      int lh = -1;
      light_test(sc, from, dir, tl, lh);
      lc.rays++;
      lc.prim += cast == B_EYE0 + CAST;
      lc.ext += cast == B_LIGHT + CAST || cast == B_EYE + CAST;
      lc.shadow += cast == TO_LIGHT;
      lc.conn += cast == TO_VERTEX;
      if (!segment) {
        ro = from;
        rd = dir;
        k = lh;
        tmax = tl;
        phase = cast - CAST;
        emit = 1;
        lc.trav++;
      } else {
        if (lh < 0) {
          out.add(bb, p, cast == TO_VERTEX ? cnt.j : 0, dir, limit);
          lc.trav++;
        } else if (cast == TO_LIGHT) {   // a light closes the segment: occluded
          const f4 em = ld4(sc.mats[e.mat].ke);
          color = color + (ev.contrib(cnt.i) * (em + (ym::splat(0.0f) + em))) * weight;
        }
        if (cast == TO_VERTEX) cnt.j -= 1;
      }
      cast = 0;
    }
    if (!__any_sync(mask, !emit && phase != Q_FINISH)) break;
  }
  if (!emit) {   // the running mean of the pixel
    if (ym::any_nan(color)) color = ym::mk(0.988f, 0.0588f, 0.7529f, 1.0f);
    const float4 prev = pp.accum[pix];
    f4 cc = color;
    if (pp.reset == 1) {
      cc.w = 1.0f;
    } else {
      const int np = (int)prev.w;
      cc = cc + f4of(prev) * (float)np;
      cc = cc / (float)(np + 1);
      cc.w = (float)(np + 1);
    }
    pp.accum[pix] = make_float4(cc.x, cc.y, cc.z, cc.w);
    lc.samples++;
  }
  if (emit) {
    ps.misc[p] = make_int4((int)seed, pix, pack_st(phase, flags & 15, lj, k), pack_cnt(cnt));
    if (conn_live) {
      ps.thr[p] = make_float4(color.x, color.y, color.z, color.w);
      ps.thr_next[p] = make_float4(sub.x, sub.y, sub.z, sub.w);
      ps.indirect[p] = make_float4(light_pdf, 0.0f, 0.0f, 0.0f);
    }
    ps.direct[p] = make_float4(weight, ks, pend_pdf, pend_prob);
    if (emit == 2) {
      ps.ro[p] = make_float4(e.hp.x, e.hp.y, e.hp.z, 0.0f);
      ps.job[p] = make_int4((int)out.js, (int)(out.js >> 32), out.n, 0);
    } else {
      ps.ro[p] = make_float4(ro.x, ro.y, ro.z, tmax);
      ps.rd[p] = make_float4(rd.x, rd.y, rd.z, rd.w);
    }
  }
  return emit == 2 ? EMIT_WAIT | (((1 << out.n) - 1) * EMIT_SEG0) : emit;
}

__global__ void __launch_bounds__(256, 2) k_logic_bdpt(PassParams pp, PathState ps, BdptBuffers bb,
                                                    const int* __restrict__ in_closest, const int* __restrict__ in_wait,
                                                    const RoundCounters* rc_in, int* out_closest, int* out_wait,
                                                    RoundCounters* rc_out, DevStats* st, const int* __restrict__ sorted,
                                                    const SortCtl* sctl) {
  __shared__ unsigned long long s_cnt[8];   // rays, primary, extension, shadow, connection, traversed, samples
  if (threadIdx.x < 8) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int nc = rc_in->n_closest, na = rc_in->n_wait;
  const int n = nc + na;
  const int lane = threadIdx.x & 31;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps_total = (gridDim.x * blockDim.x) >> 5;
  const bool use_sorted = sctl && sctl->use;

  for (int wbase = warp_global * 32; wbase < n; wbase += warps_total * 32) {
    const int entry = wbase + lane;
    int sent = 0;
    int p = -1;
    LogicCounts lc;
    const unsigned mask = __ballot_sync(0xffffffffu, entry < n);
    if (entry < n) {
      p = use_sorted ? sorted[entry] : (entry < nc ? in_closest[entry] : in_wait[entry - nc]);
      sent = bdpt_step(pp, ps, bb, p, lc, mask);
    }
    append_bdpt(bb, sent & EMIT, p, __popc(sent / EMIT_SEG0), out_closest, out_wait, rc_out);
    const unsigned c[7] = {lc.rays, lc.prim, lc.ext, lc.shadow, lc.conn, lc.trav, lc.samples};
#pragma unroll
    for (int q = 0; q < 7; ++q) {
      unsigned x = c[q];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
      if (lane == 0 && x) atomicAdd(&s_cnt[q], (unsigned long long)x);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_cnt[0]) atomicAdd(&st->rays, s_cnt[0]);
    if (s_cnt[1]) atomicAdd(&st->primary, s_cnt[1]);
    if (s_cnt[2]) atomicAdd(&st->extension, s_cnt[2]);
    if (s_cnt[3]) atomicAdd(&st->shadow, s_cnt[3]);
    if (s_cnt[4]) atomicAdd(&st->connection, s_cnt[4]);
    if (s_cnt[5]) atomicAdd(&st->traversed, s_cnt[5]);
    if (s_cnt[6]) atomicAdd(&st->samples, s_cnt[6]);
  }
}

void launch_logic_bdpt(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                       const int* in_wait, const RoundCounters* rc_in, int* out_closest, int* out_wait,
                       RoundCounters* rc_out, DevStats* st, int grid, cudaStream_t s, const int* sorted,
                       const SortCtl* sctl) {
  k_logic_bdpt<<<grid, 256, 0, s>>>(pp, ps, bb, in_closest, in_wait, rc_in, out_closest, out_wait, rc_out, st, sorted,
                                    sctl);
}

struct BdptStep {
  static constexpr bool FAN = true, BDPT = true;
  const PassParams& pp;
  const PathState& ps;
  const BdptBuffers& bb;
  __device__ __forceinline__ int segments(int p) const {
    return (ps.misc[p].z & 15) == B_FAN ? ((1 << ps.job[p].z) - 1) * EMIT_SEG0 : 0;
  }
  __device__ __forceinline__ int operator()(int p, unsigned mask, LogicCounts& lc) const {
    return bdpt_step(pp, ps, bb, p, lc, mask);
  }
};

// The tail kernel (yc_tail.cuh), which spares a pass its last rounds of few paths (each ten launches,
// most of them empty, and the latency of a walk): a 1280x720 pass over 820K triangles 9.54 -> 9.10
// ms, a 160x120 pass over 60K 2.40 -> 1.51. Two blocks per SM: the shading and the walk hold 198
// registers.
template <bool WIDE>
__global__ void __launch_bounds__(TAIL_TB, 2) k_tail_bdpt(PassParams pp, PathState ps, BdptBuffers bb,
                                                         const int* __restrict__ in_closest,
                                                         const int* __restrict__ in_wait, RoundCounters* rc_in,
                                                         int threshold, int stack_cap, DevStats* st, int n_smem,
                                                         int* spill) {
  tail_loop<WIDE>(BdptStep{pp, ps, bb}, pp.sc, ps, bb.sg, in_closest, in_wait, rc_in, threshold, stack_cap, st, n_smem,
                  spill);
}

int tail_bdpt_grid(const PassParams& pp, int n_smem) {
  const size_t smem = tail_smem(tail_entries(pp.sc.depth, n_smem));
  return pp.sc.wide ? tail_grid_of(k_tail_bdpt<true>, smem) : tail_grid_of(k_tail_bdpt<false>, smem);
}

int launch_tail_bdpt(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                     const int* in_wait, RoundCounters* rc_in, int threshold, DevStats* st, int grid, cudaStream_t s,
                     int n_smem, int* spill) {
  n_smem = tail_entries(pp.sc.depth, spill ? n_smem : 0);
  const auto kernel = pp.sc.wide ? k_tail_bdpt<true> : k_tail_bdpt<false>;
  kernel<<<grid, TAIL_TB, tail_smem(n_smem), s>>>(pp, ps, bb, in_closest, in_wait, rc_in, threshold, pp.sc.depth + 2, st,
                                                  n_smem, spill);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace yc
