// bdpt.cu -- wavefront form of Yune's naive bidirectional path tracer
// (kernels/legacy/bdpt.cl:158-640), step (f) of the pipeline.
//
// Per sample the reference builds a light subpath (createLightPath, bdpt.cl:432-511),
// an eye subpath (createEyePath, bdpt.cl:513-560), then for every eye vertex adds its
// emission and next-event estimate and connects it to every light vertex j >= 1 with a
// shadow ray (shading, bdpt.cl:562-640). Here each path is a state machine like the
// unidirectional one (udpt.cu): the logic kernel advances it to its next ray, the extend
// and occlusion kernels trace the queues, and the subpath vertices live in HBM as one
// 64-byte record per vertex (two full 32-byte sectors: a connection reads two vertices of
// a path whose neighbours in the queue are unrelated), vertex k of path p at
// [(p * bounces + k) * 4 + field]:
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

namespace yc {

enum : int { BF_GLOSSY = 1 };
constexpr int CAST = 1;   // a pending cast holds its state + CAST (0: none)

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
__global__ void __launch_bounds__(256) k_raygen_bdpt(PassParams pp, PathState ps, BdptBuffers bb, int* q_closest,
                                                     RoundCounters* rc, DevStats* st) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = pp.tile_w * pp.tile_h;
  int px = 0, py = 0;
  bool active = false;
  if (gid < n) {
    px = gid % pp.tile_w + pp.off_x;
    py = gid / pp.tile_w + pp.off_y;
    active = px < pp.width && py < pp.height;
  }
  const int W = pp.width, H = pp.height;
  const int pix = py * W + px;
  const int slot = pix;
  bool eye_first = false;
  if (active) {
    const DevScene& sc = pp.sc;
    uint32_t seed = (uint32_t)((py + 1) * W + (px + 1));
    seed = pp.rand_seed * seed;
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
    f4 d;
    d.x = ym::dot(ld4(pp.cam.r1), dir);
    d.y = ym::dot(ld4(pp.cam.r2), dir);
    d.z = ym::dot(ld4(pp.cam.r3), dir);
    d.w = ym::dot(ld4(pp.cam.r4), dir);
    d = ym::normalize(d);
    VertexRef ev{bb.ev + (size_t)slot * bb.bounces * 4};
    VertexRef lv{bb.lv + (size_t)slot * bb.bounces * 4};
    ev.at(0, 2) = make_float4(d.x, d.y, d.z, d.w);   // the camera ray, traced after the light subpath
    // light vertex 0 on light 0 (createLightPath, bdpt.cl:435-456)
    const yc_quad_light& L = sc.lights[0];
    seed = ym::xor_shift(seed);
    const float lr1 = (float)((double)seed / 4294967295.0);   // seed / (double)UINT_MAX
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
  const unsigned m = __ballot_sync(0xffffffffu, active);
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0 && m) base = atomicAdd(&rc->n_closest, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (active) q_closest[base + __popc(m & ((1u << lane) - 1))] = slot;
  const unsigned m_eye = __ballot_sync(0xffffffffu, active && eye_first);
  if (lane == 0 && m) {
    atomicAdd(&st->rays, (unsigned long long)__popc(m));
    atomicAdd(&st->traversed, (unsigned long long)__popc(m));
    if (m_eye) atomicAdd(&st->primary, (unsigned long long)__popc(m_eye));
    if (m & ~m_eye) atomicAdd(&st->extension, (unsigned long long)__popc(m & ~m_eye));
  }
}

void launch_raygen_bdpt(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, int* q_closest,
                        RoundCounters* rc, DevStats* st, cudaStream_t s) {
  const int n = pp.tile_w * pp.tile_h;
  k_raygen_bdpt<<<(n + 255) / 256, 256, 0, s>>>(pp, ps, bb, q_closest, rc, st);
}

// ---- logic: advance each path to its next ray ----
__global__ void __launch_bounds__(256) k_logic_bdpt(PassParams pp, PathState ps, BdptBuffers bb,
                                                    const int* __restrict__ in_closest, const int* __restrict__ in_any,
                                                    const RoundCounters* rc_in, int* out_closest, int* out_any,
                                                    RoundCounters* rc_out, DevStats* st, const int* __restrict__ sorted,
                                                    const SortCtl* sctl) {
  __shared__ unsigned long long s_cnt[8];   // rays, primary, extension, shadow, connection, traversed, samples
  if (threadIdx.x < 8) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int nc = rc_in->n_closest, na = rc_in->n_any;
  const int n = nc + na;
  const int lane = threadIdx.x & 31;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps_total = (gridDim.x * blockDim.x) >> 5;
  const DevScene& sc = pp.sc;
  const float INF = __int_as_float(0x7f800000);
  const int BOUNCES = bb.bounces;
  const int RR = 4;   // RR_THRESHOLD of bdpt.cl:4
  const bool use_sorted = sctl && sctl->use;

  for (int wbase = warp_global * 32; wbase < n; wbase += warps_total * 32) {
    const int entry = wbase + lane;
    int emit = 0;
    int p = -1;
    unsigned c[7] = {0, 0, 0, 0, 0, 0, 0};
    const unsigned mask = __ballot_sync(0xffffffffu, entry < n);
    if (entry < n) {
      p = use_sorted ? sorted[entry] : (entry < nc ? in_closest[entry] : in_any[entry - nc]);
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
      // fields (colour, sub-sum, NEE direction) are dead: Q_CONNECT initialises them.
      // They are loaded in the connection states only and stored once the stage has
      // started; the ray origin is read only where a hit point is built from it.
      const bool building = phase == B_LIGHT || phase == B_EYE0 || phase == B_EYE;
      bool conn_live = !building;
      f4 color = ym::splat(0.0f), sub = ym::splat(0.0f), w_i = ym::splat(0.0f);
      float light_pdf = 0.0f;
      if (!building) {
        color = f4of(ps.thr[p]);
        sub = f4of(ps.thr_next[p]);
        const float4 nee = ps.indirect[p];
        w_i = ym::mk(nee.x, nee.y, nee.z, 0.0f);
        light_pdf = nee.w;
      }
      float4 dv = ps.direct[p];
      float weight = dv.x, ks = dv.y, pend_pdf = dv.z, pend_prob = dv.w;
      f4 ro = ym::splat(0.0f), rd = ym::splat(0.0f);
      float tmax = 0.0f;
      if (building) {
        const float4 ro4 = ps.ro[p];
        ro = ym::mk(ro4.x, ro4.y, ro4.z, 1.0f);
        tmax = ro4.w;
      }
      if (building || phase == B_CONN) {
        const float4 rd4 = ps.rd[p];
        rd = ym::mk(rd4.x, rd4.y, rd4.z, rd4.w);
      }
      const float4 hit = ps.hit[p];

      // ---- the result of the ray the path waited for ----
      // Its BRDFs: at the vertex a subpath ray left, at the eye vertex of a light sample, or at
      // the eye vertex and then the light vertex of a connection; one copy of the lobe choice and
      // the BRDF for all of them.
      const bool light = phase == B_LIGHT, subpath = phase == B_LIGHT || phase == B_EYE;
      const int tri = __float_as_int(hit.w);
      const bool made = building && tri >= 0 && !(light && pend_pdf <= 0.0f);   // a vertex is made
      const bool seen = !building && hit.x == 0.0f;                             // a segment is free
      Vtx v, e;           // the vertex made; the eye vertex of the connection stage
      v.hp = v.n = e.hp = e.n = ym::splat(0.0f);
      v.mat = e.mat = 0;
      if (made) v = tri_vertex(sc, ro, rd, hit.x, hit.y, hit.z, tri);
      if (!building) e = ev.vtx(cnt.i);
      f4 f0 = ym::splat(0.0f), f1 = ym::splat(0.0f), pn = ym::splat(0.0f);
      float prob0 = 0.0f;
      __syncwarp(mask);
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        if (side == 0 ? (made && subpath && !(light && cnt.i == 1)) || seen : seen && phase == B_CONN) {
          Vtx at = e;
          f4 w_in = phase == B_NEE ? w_i : rd, w_out = ym::splat(0.0f);
          bool g = (flags & BF_GLOSSY) != 0;
          float prob = pend_prob;
          if (subpath) {
            const VertexRef& sv = light ? lv : ev;
            const f4 back = -sv.dir(cnt.i - 1);
            at = sv.vtx(cnt.i - 1);
            pn = at.n;
            w_in = light ? back : rd;
            w_out = light ? rd : back;
          } else {
            if (side) {
              at = lv.vtx(cnt.j);
              w_in = -lv.dir(cnt.j);
              w_out = -rd;
            } else {
              w_out = -ev.dir(cnt.i);
            }
            g = sample_glossy_b(sc.mats[at.mat], seed, prob);
            if (side == 0) prob0 = prob;
          }
          const f4 f = brdf_b(w_in, w_out, at.n, sc.mats[at.mat], g, prob);
          if (side) f1 = f;
          else f0 = f;
        }
        if (!__any_sync(mask, seen && phase == B_CONN)) break;
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
      } else if (phase == B_NEE) {   // bdpt.cl:662-671 (MIS off, as shipped)
        const f4 em = ld4(sc.mats[e.mat].ke);
        f4 dl = ym::splat(0.0f) + em;   // light_sample (0) + emission
        if (seen) {
          if (prob0 == 0.0f) {
            dl = em;
          } else {
            f4 ls = (f0 * ld4(sc.lights[lj].ke)) * ym::fmax(ym::dot(w_i, e.n), 0.0f);
            ls = ls * ym::div(1.0f, light_pdf);
            dl = ls + em;
          }
        }
        color = color + (ev.contrib(cnt.i) * (em + dl)) * weight;
        cnt.j = cnt.lp - 1;
        phase = Q_SEGMENTS;
      } else {   // B_CONN, bdpt.cl:616-634
        if (seen) {
          const Vtx l_v = lv.vtx(cnt.j);
          float dist = ym::length(l_v.hp - e.hp);
          dist = ym::mul(dist, dist);
          const float gf = ym::div(ym::mul(ym::max(ym::dot(rd, e.n), 0.0f), ym::max(ym::dot(-rd, l_v.n), 0.0f)), dist);
          f4 tlp = lv.contrib(cnt.j);
          tlp = tlp * ((gf * f0) * f1);
          tlp = tlp * ev.contrib(cnt.i);
          sub = sub + tlp;
        }
        cnt.j -= 1;
        phase = Q_SEGMENTS;
      }
      // ---- a subpath's next direction, from the vertex just made (bdpt.cl:473-484, 527-535) ----
      int cast = 0;           // the state the next ray will be waited for in
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
      // ---- the connection stage until its next ray ----
      // Each pass takes the path to a segment worth a ray: the light sample of an eye vertex, or
      // the next light vertex whose segment both ends face. The light loop appears once, for
      // every kind of ray; a segment a light closes sends the path round again. With one copy
      // of the stages per state (a switch that looped over rejected segments while other lanes
      // shaded) a 1280x720 pass over 758K triangles took 4.63 ms of shading, now 3.61 ms.
      for (;;) {
        __syncwarp(mask);
        if (phase == Q_VERTEX) {   // emission + next-event estimate at eye vertex i (bdpt.cl:591-597, 642-660)
          e = ev.vtx(cnt.i);
          const yc_material& m = sc.mats[e.mat];
          sub = ym::mk(0.0f, 0.0f, 0.0f, 1.0f);
          ks = ym::max(ym::max(m.ks.x, ym::max(m.ks.y, m.ks.z)), 0.1f);
          f4 wi_raw;
          lj = sample_lights(sc, e, seed, light_pdf, wi_raw);
          if (lj == -1 || light_pdf <= 0.0f) {
            color = color + (ev.contrib(cnt.i) * (ld4(m.ke) + ld4(m.ke))) * weight;   // DL = emission
            cnt.j = cnt.lp - 1;
            phase = Q_SEGMENTS;
          } else {
            limit = ym::sub(ym::length(wi_raw), ym::mul(EPS_F, 1.5f));
            w_i = ym::normalize(wi_raw);
            org = e.hp;
            dir = w_i;
            cast = B_NEE + CAST;
          }
        }
        __syncwarp(mask);
        if (phase == Q_SEGMENTS && !cast) {   // the next connection j (bdpt.cl:598-615)
          while (cnt.j > 0 && !cast) {
            const float4 h4 = lv.at(cnt.j, 0), n4 = lv.at(cnt.j, 1);
            const f4 l_hp = ym::mk(h4.x, h4.y, h4.z, 1.0f), l_n = ym::mk(n4.x, n4.y, n4.z, 0.0f);
            dir = ym::normalize(l_hp - e.hp);
            if (ym::dot(dir, e.n) <= 0.0f || ym::dot(-dir, l_n) <= 0.0f) { cnt.j -= 1; continue; }
            org = e.hp;
            limit = ym::length(l_hp - (e.hp + dir * EPS_F));
            cast = B_CONN + CAST;
          }
          if (!cast) {
            color = color + sub * ym::mul(weight, ym::sub(1.0f, ks));
            weight = ym::mul(weight, ks);
            cnt.i += 1;
            phase = cnt.i >= cnt.ep || weight == 0.0f ? Q_FINISH : Q_VERTEX;
          }
        }
        __syncwarp(mask);
        if (cast) {   // traceRay's light loop (udpt.cl:244-276)
          const int to = cast - CAST;
          const bool segment = to == B_NEE || to == B_CONN;
          ro = to == B_EYE0 ? org : org + dir * EPS_F;
          rd = dir;
          tmax = limit;
          float tl = tmax;
          int lh = -1;
          light_test(sc, ro, rd, tl, lh);
          c[0]++;
          c[1] += to == B_EYE0;
          c[2] += to == B_LIGHT || to == B_EYE;
          c[3] += to == B_NEE;
          c[4] += to == B_CONN;
          cast = 0;
          if (!segment) {
            k = lh;
            tmax = tl;
            phase = to;
            emit = 1;
          } else if (lh < 0) {
            phase = to;
            emit = 2;
          } else if (to == B_CONN) {   // a light closes the segment: occluded
            cnt.j -= 1;
          } else {
            const f4 em = ld4(sc.mats[e.mat].ke);
            color = color + (ev.contrib(cnt.i) * (em + (ym::splat(0.0f) + em))) * weight;
            cnt.j = cnt.lp - 1;
            phase = Q_SEGMENTS;
          }
          if (emit) c[5]++;
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
        c[6]++;
      }
      if (emit) {
        ps.misc[p] = make_int4((int)seed, pix, pack_st(phase, flags & 15, lj, k), pack_cnt(cnt));
        if (conn_live) {
          ps.thr[p] = make_float4(color.x, color.y, color.z, color.w);
          ps.thr_next[p] = make_float4(sub.x, sub.y, sub.z, sub.w);
          ps.indirect[p] = make_float4(w_i.x, w_i.y, w_i.z, light_pdf);
        }
        ps.direct[p] = make_float4(weight, ks, pend_pdf, pend_prob);
        ps.ro[p] = make_float4(ro.x, ro.y, ro.z, tmax);
        ps.rd[p] = make_float4(rd.x, rd.y, rd.z, rd.w);
      }
    }
    const unsigned mc = __ballot_sync(0xffffffffu, emit == 1);
    const unsigned ma = __ballot_sync(0xffffffffu, emit == 2);
    int bc = 0, ba = 0;
    if (lane == 0) {
      if (mc) bc = atomicAdd(&rc_out->n_closest, __popc(mc));
      if (ma) ba = atomicAdd(&rc_out->n_any, __popc(ma));
    }
    bc = __shfl_sync(0xffffffffu, bc, 0);
    ba = __shfl_sync(0xffffffffu, ba, 0);
    const unsigned below = (1u << lane) - 1;
    if (emit == 1) out_closest[bc + __popc(mc & below)] = p;
    if (emit == 2) out_any[ba + __popc(ma & below)] = p;
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
                       const int* in_any, const RoundCounters* rc_in, int* out_closest, int* out_any,
                       RoundCounters* rc_out, DevStats* st, int grid, cudaStream_t s, const int* sorted,
                       const SortCtl* sctl) {
  k_logic_bdpt<<<grid, 256, 0, s>>>(pp, ps, bb, in_closest, in_any, rc_in, out_closest, out_any, rc_out, st, sorted,
                                    sctl);
}

}  // namespace yc
