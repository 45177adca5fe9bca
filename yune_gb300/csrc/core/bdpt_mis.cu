// bdpt_mis.cu -- wavefront bidirectional path tracer with multiple importance sampling
// (integrator YC_BDPT_MIS).
//
// bdpt.cl stores forward and reverse densities on its vertices but never uses them; its
// connections are summed with the heuristic weight `weight * (1 - ks)` (bdpt.cl:38-39, 453,
// 465, 598-636), so it converges to another image than the unidirectional tracer. This
// integrator weights every strategy (s light vertices, t >= 2 eye vertices; no light
// tracing to the camera) with the power heuristic over the strategies that can make the
// same path. The denominators come from two partial sums per subpath vertex (the
// recursive form of Georgiev, "Implementing Vertex Connection and Merging", 2012):
// arriving at vertex v from u with solid-angle density w_f, squared distance d2 and
// cosine c_v at v,
//   r_v = (d2 / (w_f c_v))^2,   s_v = r_v (c_u / d2)^2 acc_u,
// and once v's next direction fixes its reverse density w_r, acc_v = r_v + s_v w_r^2.
// A connection of eye vertex Y to light vertex L then has the weight
//   1 / (1 + (w_{Y->L} c_L / d2)^2 (r_L + s_L w_{L,rev}^2) + (w_{L->Y} c_Y / d2)^2 (r_Y + s_Y w_{Y,rev}^2)).
// The random-number order, the material and light models and the operation order are
// those of the CPU statement the parity tests compare against; each sample is one state
// machine as in bdpt.cu (one subpath ray, or the segments of one eye vertex, in flight), with the light subpath in 64-byte vertex
// records, vertex k of path p at [(p * bounces + k) * 4 + field]:
//   field 0: hit point xyz, material index (int bits; -1 for the point on the light)
//   field 1: shading normal xyz, r
//   field 2: direction of the ray that reached the vertex xyz, s
//   field 3: subpath throughput xyz
// The eye subpath is walked vertex by vertex: next-event estimate, then the connections
// to every stored light vertex, then the next eye ray. Path slot fields:
//   thr      pixel colour              thr_next  eye throughput xyz, r of the eye vertex
//   direct   light sample's contribution if its segment is free xyz, s of the eye vertex
//   indirect throughput after the pending bounce xyz, its solid-angle density
//   ls       cosine toward the pending ray at its origin, acc of the origin vertex,
//            area density of the light subpath's start point
//   hp, nrm, wo   the current eye vertex: point + material, normal, arriving direction
//   wi       the camera ray, kept while the light subpath is traced
#include <cuda_runtime.h>

#include "yc_bdpt.h"
#include "yc_shade.cuh"
#include "yc_tail.cuh"

namespace yc {

namespace {

enum : int { M_EYE_START = 8, M_VERTEX = 9, M_CONN = 10, M_CONT = 11, M_FINISH = 12, M_LIGHT_CONT = 13 };

struct MCount {
  int j, m, nl;   // light vertex index, eye vertex index, stored light vertices
};
__device__ __forceinline__ int pack_mc(const MCount& c) { return c.j | (c.m << 6) | (c.nl << 12); }
__device__ __forceinline__ MCount unpack_mc(int v) { return MCount{v & 63, (v >> 6) & 63, (v >> 12) & 63}; }
__device__ __forceinline__ int pack_ms(int state, int lk, int k) { return state | ((lk + 1) << 8) | ((k + 1) << 13); }

__device__ __forceinline__ float mis(float x) { return ym::mul(x, x); }
// a * b with 0 * inf = 0 (a vanishing density removes the strategy)
__device__ __forceinline__ float mul0(float a, float b) { return (a == 0.0f || b == 0.0f) ? 0.0f : ym::mul(a, b); }
__device__ __forceinline__ f4 rgb(const yc_float4& c) { return ym::mk(c.x, c.y, c.z, 0.0f); }

__device__ __forceinline__ float diffuse_prob(const yc_material& m) {
  const float sd = ym::add(ym::add(m.kd.x, m.kd.y), m.kd.z);
  const float ss = ym::add(ym::add(m.ks.x, m.ks.y), m.ks.z);
  if (ss == 0.0f) return 1.0f;
  if (sd == 0.0f) return 0.0f;
  return ym::div(sd, ym::add(sd, ss));
}

__device__ __forceinline__ f4 mirror(f4 w, f4 n) { return ym::normalize(ym::mul(2.0f, ym::dot(w, n)) * n - w); }

// What a step of the weights needs at vertex v between the directions a, toward the previous
// subpath vertex, and b, toward the next one: the solid-angle densities with which
// sample_dir picks b arriving from a and a arriving from b, and the BRDF.
struct VtxEval {
  float fwd, rev;
  f4 f;
};
__device__ __forceinline__ float pdf_at(const yc_material& m, float pd, float cn, float ca) {
  if (!(cn > 0.0f)) return 0.0f;
  float p = ym::mul(pd, ym::mul(cn, INV_PI_F));
  if (pd < 1.0f) {
    const int pe = (int)ym::add(m.px, m.py);
    const float lobe = ym::mul(ym::mul(ym::mul((float)(pe + 1), 0.5f), INV_PI_F), ym::pow(ca, (float)pe));
    p = ym::add(p, ym::mul(ym::sub(1.0f, pd), lobe));
  }
  return p;
}
__device__ __forceinline__ VtxEval eval_at(const Vtx& v, const yc_material& m, f4 a, f4 b, int brdf_model,
                                           const float2* on_ab) {
  const bool glossy = ym::length3(ld4(m.ks)) != 0.0f;
  const float pd = diffuse_prob(m);
  VtxEval r;
  float c[2] = {0.0f, 0.0f};   // the lobes' cosines, of b about a's mirror direction and the other way
  if (pd < 1.0f || glossy) {
    c[0] = ym::fmax(ym::dot(b, mirror(a, v.n)), 0.0f);
    c[1] = ym::fmax(ym::dot(a, mirror(b, v.n)), 0.0f);
  }
  float p[2];
#pragma unroll 1
  for (int k = 0; k < 2; ++k) p[k] = pdf_at(m, pd, ym::dot(k ? a : b, v.n), k ? c[1] : c[0]);
  r.fwd = p[0];
  r.rev = p[1];
  if (brdf_model == 1 && !glossy) r.f = oren_nayar(b, a, v, m, on_ab[v.mat]);
  else r.f = ld4(m.kd) * INV_PI_F;
  if (glossy) {
    const float ca = ym::pow(c[0], ym::add(m.px, m.py));
    const int pe = (int)ym::add(m.px, m.py);
    r.f = r.f + (((ld4(m.ks) * ca) * (float)(pe + 2)) * INV_PI_F) * 0.5f;
  }
  r.f.w = 0.0f;
  return r;
}

// lobe (1 number), then a cosine or Phong-lobe direction (2 numbers); false when the
// direction does not leave the surface
__device__ __forceinline__ bool sample_dir(const Vtx& v, const yc_material& m, f4 w_prev, uint32_t& seed,
                                           f4& w_next) {
  const float u = draw(seed);
  const float pd = diffuse_prob(m);
  float pdf = 0.0f;
  w_next = sample_lobe_b(v, m, !(pd >= 1.0f || u < pd), w_prev, seed, pdf);
  return ym::dot(w_next, v.n) > 0.0f;
}

// picks a light (1 number) with probability proportional to (ke.r + ke.g + ke.b) * area
__device__ __forceinline__ int pick_light(const DevScene& sc, uint32_t& seed) {
  const float u = draw(seed);
  if (!(light_total(sc.lights[0]) > 0.0f)) return -1;
  float cum = 0.0f;
  int last = -1;
  for (int i = 0; i < sc.n_lights; ++i) {
    if (!(light_weight(sc.lights[i]) > 0.0f)) continue;
    last = i;
    const float p = light_share(sc.lights[i]);
    if (u < ym::add(cum, p)) return i;
    cum = ym::add(cum, p);
  }
  return last;
}
__device__ __forceinline__ f4 light_point(const yc_quad_light& L, uint32_t& seed) {
  const float a = draw(seed);
  const float b = draw(seed);
  return (ld4(L.pos) + ld4(L.edge_l) * a) + ld4(L.edge_w) * b;
}

struct MisRec {
  float4* base;   // the path's first light vertex
  __device__ __forceinline__ float4& at(int k, int f) const { return base[(size_t)k * 4 + f]; }
  __device__ __forceinline__ Vtx vtx(int k) const {
    const float4 a = at(k, 0), b = at(k, 1);
    Vtx v;
    v.hp = ym::mk(a.x, a.y, a.z, 1.0f);
    v.n = ym::mk(b.x, b.y, b.z, 0.0f);
    v.mat = __float_as_int(a.w);
    return v;
  }
};

}  // namespace

// ---- raygen: pixel prologue, camera ray kept, light point and the first light ray ----
__global__ void __launch_bounds__(256) k_raygen_bdpt_mis(PassParams pp, int n, int row, PathState ps,
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
    ps.wi[slot] = make_float4(d.x, d.y, d.z, d.w);
    const MisRec lv{bb.lv + (size_t)slot * bb.bounces * 4};
    const int lk = pick_light(sc, seed);
    f4 o = ym::mk(pp.cam.r1.w, pp.cam.r2.w, pp.cam.r3.w, pp.cam.r4.w), rdir = d;
    int state = B_EYE0;
    MCount cnt{0, 0, 0};
    float p0 = 0.0f, c0 = 0.0f;
    if (lk >= 0) {
      const yc_quad_light& L = sc.lights[lk];
      p0 = light_point_pdf(L);
      Vtx v0;
      v0.hp = light_point(L, seed);
      v0.n = ld4(L.normal);
      v0.mat = -1;
      lv.at(0, 0) = make_float4(v0.hp.x, v0.hp.y, v0.hp.z, __int_as_float(-1));
      lv.at(0, 1) = make_float4(v0.n.x, v0.n.y, v0.n.z, 0.0f);
      float pdf = 0.0f;
      const f4 ldir = sample_cosine(v0, seed, pdf);
      c0 = ym::dot(ldir, v0.n);
      if (c0 > 0.0f) {
        o = v0.hp + ldir * EPS_F;
        rdir = ldir;
        state = B_LIGHT;
        cnt.j = 1;
      }
    }
    eye_first = state == B_EYE0;
    float len = __int_as_float(0x7f800000);
    int k = -1;
    light_test(sc, o, rdir, len, k);
    ps.misc[slot] = make_int4((int)seed, pix, pack_ms(state, lk, k), pack_mc(cnt));
    ps.ro[slot] = make_float4(o.x, o.y, o.z, len);
    ps.rd[slot] = make_float4(rdir.x, rdir.y, rdir.z, rdir.w);
    ps.indirect[slot] = make_float4(1.0f, 1.0f, 1.0f, ym::mul(c0, INV_PI_F));
    ps.ls[slot] = make_float4(c0, lk >= 0 ? ym::div(1.0f, mis(p0)) : 0.0f, p0, 0.0f);
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

void launch_raygen_bdpt_mis(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, int* q_closest,
                            RoundCounters* rc, DevStats* st, cudaStream_t s) {
  const int n = tile_pixels(pp);
  if (n > 0) k_raygen_bdpt_mis<<<(n + 255) / 256, 256, 0, s>>>(pp, n, tile_row(pp), ps, bb, q_closest, rc, st);
}

// ---- logic: advance each path to its next ray ----
// Bound by the latency of a long dependent chain at few warps: 168 registers in three blocks
// of 128 per SM measured best (unbounded, 210 in two: 2.98 ms per two 512x512 passes; three:
// 2.70; four, 386 B spilled: 2.87; five, 768 B: 3.22).
constexpr int MIS_TB = 128;
constexpr int TO_LIGHT = 1, TO_VERTEX = 2;   // a segment's kind
// One step of path p: from the results of its last rays until it needs new ones. Returns what it
// sends (EMIT_*), or 0 (the path has ended). `mask`: the lanes of the warp that make the call together.
__device__ __forceinline__ int bdpt_mis_step(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, int p,
                                         LogicCounts& lc, unsigned mask) {
  const DevScene& sc = pp.sc;
  const float INF = __int_as_float(0x7f800000);
  const int KMAX = bb.bounces;
  const int RR = pp.rr_threshold;
  int emit = 0;
  FanOut out;   // the segments to send
  const MisRec lv{bb.lv + (size_t)p * bb.bounces * 4};
  const int4 misc = ps.misc[p];
  uint32_t seed = (uint32_t)misc.x;
  const int pix = misc.y;
  int phase = misc.z & 15;
  const int lk = ((misc.z >> 8) & 31) - 1;
  int k = ((misc.z >> 13) & 31) - 1;
  MCount cnt = unpack_mc(misc.w);
  // only the fields the state reads are loaded, and only the changed ones are
  // written back: the eye vertex and colour exist from B_EYE on, the pending
  // bounce (throughput, density, cosine, acc) is read when its ray returns, and a
  // shadow ray's own origin and direction are not needed after it is traced
  const bool eye_state = phase >= B_EYE;
  const bool pending = phase == B_LIGHT || phase == B_EYE;
  const bool shadow = phase == B_FAN;
  const float4 l4 = ps.ls[p];
  float c_out = l4.x, acc = l4.y;
  const float p0 = l4.z;
  f4 color = ym::splat(0.0f), beta = ym::splat(0.0f), pend = ym::splat(0.0f), bnext = ym::splat(0.0f);
  float r_y = 0.0f, s_y = 0.0f, w_f = 0.0f;
  Vtx y;
  y.hp = ym::splat(0.0f);
  y.n = ym::splat(0.0f);
  y.mat = 0;
  f4 wp = ym::splat(0.0f);
  if (eye_state) {
    color = f4of(ps.thr[p]);
    const float4 tn = ps.thr_next[p], dc = ps.direct[p];
    beta = ym::mk(tn.x, tn.y, tn.z, 0.0f);
    r_y = tn.w;
    s_y = dc.w;
    pend = ym::mk(dc.x, dc.y, dc.z, 0.0f);
    const float4 a = ps.hp[p], b = ps.nrm[p], w = ps.wo[p];
    y.hp = ym::mk(a.x, a.y, a.z, 1.0f);
    y.n = ym::mk(b.x, b.y, b.z, 0.0f);
    y.mat = __float_as_int(a.w);
    wp = ym::mk(-w.x, -w.y, -w.z, -0.0f);
  }
  if (pending) {
    const float4 ind = ps.indirect[p];
    bnext = ym::mk(ind.x, ind.y, ind.z, 0.0f);
    w_f = ind.w;
  }
  f4 ro = ym::splat(0.0f), rd = ym::splat(0.0f);
  float tmax = 0.0f;
  if (!shadow) {
    const float4 ro4 = ps.ro[p], rd4 = ps.rd[p];
    ro = ym::mk(ro4.x, ro4.y, ro4.z, 1.0f);
    rd = ym::mk(rd4.x, rd4.y, rd4.z, rd4.w);
    tmax = ro4.w;
  }
  const float4 hit = ps.hit[p];
  bool moved = false;    // the eye vertex changed
  bool w_color = false, w_eye = false, w_pend = false, w_bounce = false;   // fields to write back

  // ---- the result of the ray the path waited for ----
  Vtx x;                        // the light vertex just made, where the light subpath goes on
  x.hp = x.n = ym::splat(0.0f);
  x.mat = 0;
  f4 lp = ym::splat(0.0f);      // toward the vertex before it
  float r_x = 0.0f, s_x = 0.0f;
  FanIn fan{0, 0};              // the free segments to light vertices
  if (shadow) {
    fan.load(ps.job[p], misc);
    w_color = fan.free != 0;
    if (fan.vertex(0) == 0 && (fan.free & 1u)) {   // the light sample
      color = color + pend;
      fan.free &= ~1u;
    }
    phase = M_CONN;
  } else {
    const int tri = __float_as_int(hit.w);
    const bool eye0 = phase == B_EYE0, light = phase == B_LIGHT;
    const bool met = tri >= 0;
    if (met) x = tri_vertex(sc, ro, rd, hit.x, hit.y, hit.z, tri);
    lp = -rd;
    const float cv = ym::dot(lp, x.n);   // (-dot(rd, n), and dot(-rd, n) for the camera ray: the same bits)
    const bool faces = met && cv > 0.0f;
    if (faces && !eye0) {
      const Vtx pv = light ? lv.vtx(cnt.j - 1) : y;
      const f4 dv = x.hp - pv.hp;
      const float d2 = ym::dot(dv, dv);
      r_x = mis(ym::div(d2, ym::mul(w_f, cv)));
      s_x = mul0(ym::mul(r_x, mis(ym::div(c_out, d2))), acc);
    }
    if (light) {   // light vertex j reached (or the light subpath ends)
      phase = M_EYE_START;
      if (faces) {
        const int j = cnt.j;
        lv.at(j, 0) = make_float4(x.hp.x, x.hp.y, x.hp.z, __int_as_float(x.mat));
        lv.at(j, 1) = make_float4(x.n.x, x.n.y, x.n.z, r_x);
        lv.at(j, 2) = make_float4(rd.x, rd.y, rd.z, s_x);
        lv.at(j, 3) = make_float4(bnext.x, bnext.y, bnext.z, 0.0f);
        cnt.nl = j;
        if (j + 1 <= KMAX - 2) phase = M_LIGHT_CONT;
      }
    } else if (faces) {   // an eye vertex: the first one, or vertex m + 1
      beta = eye0 ? ym::mk(1.0f, 1.0f, 1.0f, 0.0f) : bnext;
      r_y = r_x;
      s_y = s_x;
      cnt.m = eye0 ? 1 : cnt.m + 1;
      if (eye0) color = ym::mk(0.0f, 0.0f, 0.0f, 1.0f);
      y = x;
      wp = lp;
      moved = w_eye = w_pend = true;
      phase = M_VERTEX;
    } else {
      phase = M_FINISH;
      if (eye0) {
        if (met) {
          color = ym::mk(0.0f, 0.0f, 0.0f, 1.0f);
        } else if (k >= 0) {
          color = (ym::dot(rd, ld4(sc.lights[k].normal)) < 0.0f) ? ym::mk(1.0f, 1.0f, 1.0f, 1.0f)
                                                                 : ym::mk(0.1f, 0.1f, 0.1f, 1.0f);
        } else {
          color = ym::mk(0.4f, 0.4f, 0.4f, 1.0f);
        }
      } else if (!met && k >= 0) {   // the eye subpath met a light (strategy s = 0)
        const yc_quad_light& L = sc.lights[k];
        const float cl = -ym::dot(rd, ld4(L.normal));
        if (cl > 0.0f) {
          const f4 z = ro + rd * tmax;
          const f4 dv = z - y.hp;
          const float d2 = ym::dot(dv, dv);
          const float r2 = mis(ym::div(d2, ym::mul(w_f, cl)));
          const float s2 = mul0(ym::mul(r2, mis(ym::div(c_out, d2))), acc);
          const float es = ym::mul(mis(light_point_pdf(L)), ym::add(r2, mul0(s2, mis(ym::mul(cl, INV_PI_F)))));
          const float w = ym::div(1.0f, ym::add(1.0f, es));
          color = color + (bnext * rgb(L.ke)) * w;
        }
      }
    }
  }
  // ---- an eye vertex's emission, and its light sample ----
  int cand = 0;             // a segment to send: TO_LIGHT or TO_VERTEX
  f4 dir = ym::splat(0.0f); //   its direction, squared length, length and end cosines
  float d2 = 0.0f, dist = 0.0f, cy = 0.0f, cl = 0.0f, pk = 0.0f;
  int at = 0;               //   the light, or the light vertex, at its end
  __syncwarp(mask);
  if (phase == M_VERTEX) {
    color = color + beta * rgb(sc.mats[y.mat].ke);
    w_color = true;
    if (cnt.m + 1 > KMAX) {
      phase = M_FINISH;
    } else if (lk < 0) {
      phase = M_CONT;
    } else {
      cnt.j = 1;
      phase = M_CONN;
      at = pick_light(sc, seed);
      if (at >= 0) {
        const yc_quad_light& L = sc.lights[at];
        pk = light_point_pdf(L);
        const f4 v = light_point(L, seed) - y.hp;
        d2 = ym::dot(v, v);
        dist = ym::sqrt(d2);
        dir = v * ym::rcp(dist);
        cy = ym::dot(dir, y.n);
        cl = -ym::dot(dir, ld4(L.normal));
        if (cy > 0.0f && cl > 0.0f) cand = TO_LIGHT;
      }
    }
  }
  // Each pass over the stages below takes the path one step on: a free connection is
  // evaluated, a segment of the eye vertex is collected, or the subpath's next direction is
  // drawn. The evaluation at a vertex (two densities and the BRDF), which is most of the
  // work, appears once, for the light sample, both ends of a connection and the new
  // directions alike, so that lanes in different states run it together, and the segments
  // of an eye vertex are traced in one round, before the connections are evaluated (no
  // random number is drawn between them): only the free ones are. Two 512x512 passes of
  // the four-light Cornell box took 84 rounds and 6.4 ms with one segment a round, 48 and
  // 4.9 ms with eight (trace 2.44 -> 1.69 ms, shading 2.69 -> 2.34).
  // With one copy of the stages per state and the evaluation in called functions the kernel
  // ran 8-9 of 32 lanes (loops over rejected segments among them) at 195 registers: 5.75 ms
  // of shading.
  for (;;) {
    __syncwarp(mask);
    const bool conn = fan.free != 0;
    if (conn) {   // the next connection
      const int sg = __ffs(fan.free) - 1;
      fan.free &= fan.free - 1u;
      at = fan.vertex(sg);
      const float4 h4 = lv.at(at, 0), n4 = lv.at(at, 1), s4 = bb.seg[((size_t)p << bb.sg.shift) + sg];
      const f4 v = ym::mk(h4.x, h4.y, h4.z, 1.0f) - y.hp;
      d2 = ym::dot(v, v);
      dir = ym::mk(s4.x, s4.y, s4.z, 0.0f);
      cy = ym::dot(dir, y.n);
      cl = -ym::dot(dir, ym::mk(n4.x, n4.y, n4.z, 0.0f));
    } else if (phase == M_CONN && !cand) {   // the next light vertex both ends of whose segment face each other
      while (cnt.j <= cnt.nl && cnt.m + cnt.j + 1 <= KMAX && !cand && !out.full(bb)) {
        at = cnt.j++;
        const float4 h4 = lv.at(at, 0), n4 = lv.at(at, 1);
        const f4 v = ym::mk(h4.x, h4.y, h4.z, 1.0f) - y.hp;
        d2 = ym::dot(v, v);
        dist = ym::sqrt(d2);
        dir = v * ym::rcp(dist);
        cy = ym::dot(dir, y.n);
        cl = -ym::dot(dir, ym::mk(n4.x, n4.y, n4.z, 0.0f));
        if (cy > 0.0f && cl > 0.0f) cand = TO_VERTEX;
      }
      if (!cand) {
        phase = out.n > 0 ? (int)B_FAN : (int)M_CONT;
        if (out.n > 0) emit = 2;
      }
    }
    __syncwarp(mask);
    const bool light = phase == M_LIGHT_CONT;
    bool go = light || (phase == M_CONT && !emit);   // a subpath's next direction is drawn
    f4 cont = light ? bnext : beta;
    if (go) {
      const Vtx v = light ? x : y;
      if ((light ? cnt.j : cnt.m) > RR) {
        const float q = ym::min(luminance(cont), 0.95f);
        go = draw(seed) < q;
        if (go) cont = cont / q;
      }
      if (go) go = sample_dir(v, sc.mats[v.mat], light ? lp : wp, seed, dir);
      if (!go) phase = light ? M_EYE_START : M_FINISH;
    }
    __syncwarp(mask);
    // at the vertex: of a segment y, then for a connection the light vertex; of a new
    // direction the vertex it leaves
    VtxEval ev{0.0f, 0.0f, ym::splat(0.0f)}, el{0.0f, 0.0f, ym::splat(0.0f)};
    Vtx lx = x;
    float lr = 0.0f, lsv = 0.0f;
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      if (side == 0 ? conn || cand == TO_LIGHT || go : conn) {
        f4 a = light ? lp : wp, b = dir;
        Vtx v = light ? x : y;
        if (side) {
          const float4 f2 = lv.at(at, 2);
          v = lv.vtx(at);
          lr = lv.at(at, 1).w;
          lsv = f2.w;
          a = ym::mk(-f2.x, -f2.y, -f2.z, -0.0f);
          b = -dir;
        }
        const VtxEval r = eval_at(v, sc.mats[v.mat], a, b, pp.brdf_model, sc.on_ab);
        if (side) el = r;
        else ev = r;
      }
      if (!__any_sync(mask, conn)) break;
    }
    if (conn || cand == TO_LIGHT) {
      float ls, es, g;
      f4 c3;
      if (conn) {
        ls = mul0(mis(ym::div(ym::mul(ev.fwd, cl), d2)), ym::add(lr, mul0(lsv, mis(el.rev))));
        es = mul0(mis(ym::div(ym::mul(el.fwd, cy), d2)), ym::add(r_y, mul0(s_y, mis(ev.rev))));
        g = ym::div(ym::mul(cy, cl), d2);
        const float4 f3 = lv.at(at, 3);
        const f4 le = rgb(sc.lights[lk].ke) * ym::div(PI_F, p0);
        c3 = (((beta * ev.f) * el.f) * ym::mk(f3.x, f3.y, f3.z, 0.0f)) * le;
      } else {
        ls = mis(ym::div(ym::mul(ev.fwd, cl), ym::mul(d2, pk)));
        es = mul0(mis(ym::div(ym::mul(ym::mul(cl, INV_PI_F), cy), d2)), ym::add(r_y, mul0(s_y, mis(ev.rev))));
        g = ym::div(ym::mul(cy, cl), ym::mul(d2, pk));
        c3 = (beta * ev.f) * rgb(sc.lights[at].ke);
      }
      const float w = ym::div(1.0f, ym::add(ym::add(1.0f, ls), es));
      const f4 part = c3 * ym::mul(g, w);
      if (conn) color = color + part;
      else pend = part;
    } else if (go) {
      if (ev.fwd > 0.0f) {
        const Vtx v = light ? x : y;
        w_f = ev.fwd;
        c_out = ym::dot(dir, v.n);
        acc = ym::add(light ? r_x : r_y, mul0(light ? s_x : s_y, mis(ev.rev)));
        bnext = ((cont * ev.f) * c_out) / w_f;
        w_bounce = true;
      } else {
        go = false;
        phase = light ? M_EYE_START : M_FINISH;
      }
    }
    // the ray: its light loop, and whether the hierarchy has to settle it
    __syncwarp(mask);
    const bool start = phase == M_EYE_START && !emit;   // the camera ray
    if (cand || go || start) {
      ro = (light && go ? x.hp : y.hp) + dir * EPS_F;
      rd = dir;
      tmax = INF;
      if (start) {
        const float4 d = ps.wi[p];
        ro = ym::mk(pp.cam.r1.w, pp.cam.r2.w, pp.cam.r3.w, pp.cam.r4.w);
        rd = ym::mk(d.x, d.y, d.z, d.w);
        cnt.m = 0;
      } else if (cand) {
        tmax = ym::sub(dist, ym::mul(EPS_F, cand == TO_VERTEX ? 2.0f : 1.5f));
      }
      float tl = tmax;
      int lh = -1;
      light_test(sc, ro, rd, tl, lh);
      lc.rays++;
      lc.prim += start;
      lc.ext += go;
      lc.shadow += cand == TO_LIGHT;
      lc.conn += cand == TO_VERTEX;
      if (!cand) {
        k = lh;
        tmax = tl;
        if (go && light) ++cnt.j;
        phase = start ? B_EYE0 : light ? B_LIGHT : B_EYE;
        emit = 1;
      } else if (lh < 0) {   // (a light that closes the segment occludes it)
        out.add(bb, p, cand == TO_VERTEX ? at : 0, dir, tmax);
      }
      if (!cand || lh < 0) lc.trav++;
      cand = 0;
    }
    if (!__any_sync(mask, !emit && phase != M_FINISH)) break;
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
    ps.misc[p] = make_int4((int)seed, pix, pack_ms(phase, lk, k), pack_mc(cnt));
    if (w_color) ps.thr[p] = make_float4(color.x, color.y, color.z, color.w);
    if (w_eye) ps.thr_next[p] = make_float4(beta.x, beta.y, beta.z, r_y);
    if (w_pend) ps.direct[p] = make_float4(pend.x, pend.y, pend.z, s_y);
    if (w_bounce) {
      ps.indirect[p] = make_float4(bnext.x, bnext.y, bnext.z, w_f);
      ps.ls[p] = make_float4(c_out, acc, p0, 0.0f);
    }
    if (moved) {
      ps.hp[p] = make_float4(y.hp.x, y.hp.y, y.hp.z, __int_as_float(y.mat));
      ps.nrm[p] = make_float4(y.n.x, y.n.y, y.n.z, 0.0f);
      ps.wo[p] = make_float4(-wp.x, -wp.y, -wp.z, 0.0f);
    }
    if (emit == 2) {
      ps.ro[p] = make_float4(y.hp.x, y.hp.y, y.hp.z, 0.0f);
      ps.job[p] = make_int4((int)out.js, (int)(out.js >> 32), out.n, 0);
    } else {
      ps.ro[p] = make_float4(ro.x, ro.y, ro.z, tmax);
      ps.rd[p] = make_float4(rd.x, rd.y, rd.z, rd.w);
    }
  }
  return emit == 2 ? EMIT_WAIT | (((1 << out.n) - 1) * EMIT_SEG0) : emit;
}

__global__ void __launch_bounds__(MIS_TB, 3) k_logic_bdpt_mis(PassParams pp, PathState ps, BdptBuffers bb,
                                                        const int* __restrict__ in_closest,
                                                        const int* __restrict__ in_wait, const RoundCounters* rc_in,
                                                        int* out_closest, int* out_wait, RoundCounters* rc_out,
                                                        DevStats* st, const int* __restrict__ sorted,
                                                        const SortCtl* sctl) {
  // per-warp counts of rays, primary, extension, shadow, connection, traversed, samples,
  // added to the device counters when the warp leaves (no block barrier: warps finish at
  // different times)
  unsigned w_cnt[7] = {0, 0, 0, 0, 0, 0, 0};
  const int nc = rc_in->n_closest, na = rc_in->n_wait;
  const int n = nc + na;
  const int lane = threadIdx.x & 31;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps_total = (gridDim.x * blockDim.x) >> 5;
  const bool use_sorted = sctl && sctl->use;

  for (int wbase = warp_global * 32; wbase < n; wbase += warps_total * 32) {
    const int e = wbase + lane;
    int sent = 0;
    int p = -1;
    LogicCounts lc;
    const unsigned mask = __ballot_sync(0xffffffffu, e < n);
    if (e < n) {
      p = use_sorted ? sorted[e] : (e < nc ? in_closest[e] : in_wait[e - nc]);
      sent = bdpt_mis_step(pp, ps, bb, p, lc, mask);
    }
    append_bdpt(bb, sent & EMIT, p, __popc(sent / EMIT_SEG0), out_closest, out_wait, rc_out);
    const unsigned c[7] = {lc.rays, lc.prim, lc.ext, lc.shadow, lc.conn, lc.trav, lc.samples};
#pragma unroll
    for (int q = 0; q < 7; ++q) w_cnt[q] += c[q];
  }
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    unsigned x = w_cnt[q];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    w_cnt[q] = x;
  }
  if (lane == 0) {
    if (w_cnt[0]) atomicAdd(&st->rays, (unsigned long long)w_cnt[0]);
    if (w_cnt[1]) atomicAdd(&st->primary, (unsigned long long)w_cnt[1]);
    if (w_cnt[2]) atomicAdd(&st->extension, (unsigned long long)w_cnt[2]);
    if (w_cnt[3]) atomicAdd(&st->shadow, (unsigned long long)w_cnt[3]);
    if (w_cnt[4]) atomicAdd(&st->connection, (unsigned long long)w_cnt[4]);
    if (w_cnt[5]) atomicAdd(&st->traversed, (unsigned long long)w_cnt[5]);
    if (w_cnt[6]) atomicAdd(&st->samples, (unsigned long long)w_cnt[6]);
  }
}

void launch_logic_bdpt_mis(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                           const int* in_wait, const RoundCounters* rc_in, int* out_closest, int* out_wait,
                           RoundCounters* rc_out, DevStats* st, int grid, cudaStream_t s, const int* sorted,
                           const SortCtl* sctl) {
  // (grid counts blocks of 256)
  k_logic_bdpt_mis<<<grid * (256 / MIS_TB), MIS_TB, 0, s>>>(pp, ps, bb, in_closest, in_wait, rc_in, out_closest, out_wait,
                                                            rc_out, st, sorted, sctl);
}

struct BdptMisStep {
  static constexpr bool FAN = true, BDPT = true;
  const PassParams& pp;
  const PathState& ps;
  const BdptBuffers& bb;
  __device__ __forceinline__ int segments(int p) const {
    return (ps.misc[p].z & 15) == B_FAN ? ((1 << ps.job[p].z) - 1) * EMIT_SEG0 : 0;
  }
  __device__ __forceinline__ int operator()(int p, unsigned mask, LogicCounts& lc) const {
    return bdpt_mis_step(pp, ps, bb, p, lc, mask);
  }
};

// The tail kernel (yc_tail.cuh), which spares a pass its last rounds of few paths (each ten launches,
// most of them empty, and the latency of a walk): a 1280x720 pass over 820K triangles 7.69 -> 6.90
// ms, a 96x64 pass of the Cornell box 1.21 -> 0.78. Two blocks per SM: the shading and the walk hold
// 231 registers.
template <bool WIDE>
__global__ void __launch_bounds__(TAIL_TB, 2) k_tail_bdpt_mis(PassParams pp, PathState ps, BdptBuffers bb,
                                                         const int* __restrict__ in_closest,
                                                         const int* __restrict__ in_wait, RoundCounters* rc_in,
                                                         int threshold, int stack_cap, DevStats* st, int n_smem,
                                                         int* spill) {
  tail_loop<WIDE>(BdptMisStep{pp, ps, bb}, pp.sc, ps, bb.sg, in_closest, in_wait, rc_in, threshold, stack_cap, st, n_smem,
                  spill);
}

int tail_bdpt_mis_grid(const PassParams& pp, int n_smem) {
  const size_t smem = tail_smem(tail_entries(pp.sc.depth, n_smem));
  return pp.sc.wide ? tail_grid_of(k_tail_bdpt_mis<true>, smem) : tail_grid_of(k_tail_bdpt_mis<false>, smem);
}

int launch_tail_bdpt_mis(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                     const int* in_wait, RoundCounters* rc_in, int threshold, DevStats* st, int grid, cudaStream_t s,
                     int n_smem, int* spill) {
  n_smem = tail_entries(pp.sc.depth, spill ? n_smem : 0);
  const auto kernel = pp.sc.wide ? k_tail_bdpt_mis<true> : k_tail_bdpt_mis<false>;
  kernel<<<grid, TAIL_TB, tail_smem(n_smem), s>>>(pp, ps, bb, in_closest, in_wait, rc_in, threshold, pp.sc.depth + 2, st,
                                                  n_smem, spill);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace yc
