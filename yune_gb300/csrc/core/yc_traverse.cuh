// yc_traverse.cuh -- BVH traversal for sm_103a: while-while depth-first walk over the
// repacked two-child or four-child nodes with a per-thread stack in shared memory.
//
// The tests themselves are the reference's, operation for operation, so the accepted
// triangles and their t are bit-identical to traverseBVH + rayTriangleIntersection
// (kernels/legacy/udpt.cl:288-390). What changes is the order of the walk: the
// reference visits, breadth first, every box the ray's half-line crosses and keeps the
// first triangle with the smallest t; here the nearer child is visited first and a
// child is skipped once its entry distance lies beyond the closest hit found so far (by
// a margin of 2^-10 relative, so rounding of the entry distance can never hide a
// triangle the reference would accept). Between triangles at exactly the same t the
// reference keeps the first it visits; every stream slot carries that visiting rank and
// an equal-t candidate replaces the current one only when its rank is lower, so the
// closest triangle and its t are the reference's bit for bit.
//
// The translation unit is compiled with -fmad=false: no multiply-add is fused, as in
// the reference arithmetic.
#pragma once

#include <cooperative_groups.h>
#include <stdint.h>

#include "yc_scene.h"

namespace yc {

struct RayIn {
  float ox, oy, oz, tmax;
  float dx, dy, dz;
};

struct HitOut {
  float t, u, v;
  int tri;   // original triangle index, -1 when nothing closer than tmax
};

// work done by walks: child boxes tested (two per two-child node, four per four-child
// node) and triangles tested
struct WalkCount {
  unsigned nodes = 0, tris = 0;
};

// ---- packed pairs: the f32x2 operations of sm_100 and later apply the IEEE
// round-to-nearest operation to each 32-bit half of a 64-bit register, so one packed
// operation gives exactly the bits of the two scalar operations it replaces, at one
// instruction issue. The two-child node stores its bounds as (child 0, child 1) pairs.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void up2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ float lo2(f32x2 v) {
  float a, b;
  up2(v, a, b);
  return a;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// OpenCL `min` (y if y < x, otherwise x); NaN-sensitive like the reference.
__device__ __forceinline__ float ocl_min(float x, float y) { return (y < x) ? y : x; }
// OpenCL `fmax` (NaN operand ignored; ties keep x).
__device__ __forceinline__ float ocl_fmax(float x, float y) {
  if (x != x) return y;
  if (y != y) return x;
  return (x < y) ? y : x;
}

// rayAabbIntersection (udpt.cl:392-431) exactly, for rays with a zero or subnormal
// direction component (1/d = inf can make (p - o) * inv NaN, and the reference then
// skips that axis). Returns hit and the entry distance.
__device__ __forceinline__ bool box_ref(float ox, float oy, float oz, float ix, float iy, float iz,
                                        float lx, float hx, float ly, float hy, float lz, float hz,
                                        float& tentry) {
  float t_max = __int_as_float(0x7f800000), t_min = -__int_as_float(0x7f800000);
  float mn = __fmul_rn(__fsub_rn(lx, ox), ix), mx = __fmul_rn(__fsub_rn(hx, ox), ix);
  if (!(mn != mn)) { t_min = ocl_fmax(ocl_min(mn, mx), t_min); t_max = ocl_min(ocl_fmax(mn, mx), t_max); }
  mn = __fmul_rn(__fsub_rn(ly, oy), iy); mx = __fmul_rn(__fsub_rn(hy, oy), iy);
  if (!(mn != mn)) { t_min = ocl_fmax(ocl_min(mn, mx), t_min); t_max = ocl_min(ocl_fmax(mn, mx), t_max); }
  if (t_max < t_min) { tentry = t_min; return false; }
  mn = __fmul_rn(__fsub_rn(lz, oz), iz); mx = __fmul_rn(__fsub_rn(hz, oz), iz);
  if (!(mn != mn)) { t_min = ocl_fmax(ocl_min(mn, mx), t_min); t_max = ocl_min(ocl_fmax(mn, mx), t_max); }
  tentry = t_min;
  return t_max > ocl_fmax(t_min, 0.0f);
}

// rayAabbIntersection on the slab values a = (lo - o) * inv and b = (hi - o) * inv of each
// axis (computed by the caller, possibly two boxes at a time with packed operations):
// box_ref's NaN-skipping arithmetic
__device__ __forceinline__ bool box_ref_ab(float ax, float bx, float ay, float by, float az, float bz,
                                           float& tentry) {
  float t_max = __int_as_float(0x7f800000), t_min = -__int_as_float(0x7f800000);
  if (!(ax != ax)) { t_min = ocl_fmax(ocl_min(ax, bx), t_min); t_max = ocl_min(ocl_fmax(ax, bx), t_max); }
  if (!(ay != ay)) { t_min = ocl_fmax(ocl_min(ay, by), t_min); t_max = ocl_min(ocl_fmax(ay, by), t_max); }
  if (t_max < t_min) { tentry = t_min; return false; }
  if (!(az != az)) { t_min = ocl_fmax(ocl_min(az, bz), t_min); t_max = ocl_min(ocl_fmax(az, bz), t_max); }
  tentry = t_min;
  return t_max > ocl_fmax(t_min, 0.0f);
}

// minimum and maximum of three (the three-operand PTX forms of sm_100 measured no
// faster here)
__device__ __forceinline__ float max3f(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }
__device__ __forceinline__ float min3f(float a, float b, float c) { return fminf(fminf(a, b), c); }

// The same test when every 1/d is finite: no operand can be NaN, so min/max are the
// hardware FMNMX, and the reference's result is t_max > max(t_min, 0). The distance
// cull is folded in: `cull_up` is the smallest float above the cull bound (+inf when
// there is none), so min(t_max, cull_up) > max(t_min, 0) holds exactly when the box is
// hit and its entry distance is within the bound (a negative t_min, an origin inside
// the box, is never culled). tentry, which orders the children, is max(t_min, 0) when
// `clamp` (closest-hit walks: children around the origin tie and keep their order, which
// measured fewer triangle tests) and t_min otherwise (any-hit walks: the child reaching
// furthest behind the origin first, which measured fewer box tests).
__device__ __forceinline__ bool box_fast(float ox, float oy, float oz, float ix, float iy, float iz,
                                         float lx, float hx, float ly, float hy, float lz, float hz,
                                         float cull_up, bool clamp, float& tentry) {
  const float ax = __fmul_rn(__fsub_rn(lx, ox), ix), bx = __fmul_rn(__fsub_rn(hx, ox), ix);
  const float ay = __fmul_rn(__fsub_rn(ly, oy), iy), by = __fmul_rn(__fsub_rn(hy, oy), iy);
  const float az = __fmul_rn(__fsub_rn(lz, oz), iz), bz = __fmul_rn(__fsub_rn(hz, oz), iz);
  const float t0 = max3f(fminf(ax, bx), fminf(ay, by), fminf(az, bz));
  const float t1 = min3f(fmaxf(ax, bx), fmaxf(ay, by), fminf(fmaxf(az, bz), cull_up));
  const float t0c = fmaxf(t0, 0.0f);
  tentry = clamp ? t0c : t0;
  return t1 > t0c;
}

// box_fast on slab values (see box_ref_ab)
__device__ __forceinline__ bool box_fast_ab(float ax, float bx, float ay, float by, float az, float bz,
                                            float cull_up, bool clamp, float& tentry) {
  const float t0 = max3f(fminf(ax, bx), fminf(ay, by), fminf(az, bz));
  const float t1 = min3f(fmaxf(ax, bx), fmaxf(ay, by), fminf(fmaxf(az, bz), cull_up));
  const float t0c = fmaxf(t0, 0.0f);
  tentry = clamp ? t0c : t0;
  return t1 > t0c;
}

struct TriHit {
  float t, u, v;
};

// rayTriangleIntersection (udpt.cl:326-390): Moller-Trumbore with the reference's
// operation order; the `+ 0.0f` is the w-lane product of the float4 dot (0 * 0), which
// only turns a -0 sum into +0, as the reference's four-lane dot does.
__device__ __forceinline__ bool tri_test(float ox, float oy, float oz, float dx, float dy, float dz,
                                         const float4& a, const float4& b, const float4& c, float best,
                                         int best_rank, TriHit& out) {
  // e1 = b.xyz, e2 = c.xyz, v1 = a.xyz
  const float px = __fsub_rn(__fmul_rn(dy, c.z), __fmul_rn(dz, c.y));
  const float py = __fsub_rn(__fmul_rn(dz, c.x), __fmul_rn(dx, c.z));
  const float pz = __fsub_rn(__fmul_rn(dx, c.y), __fmul_rn(dy, c.x));
  const float det = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(b.x, px), __fmul_rn(b.y, py)), __fmul_rn(b.z, pz)), 0.0f);
  const float inv_det = __frcp_rn(det);
  const float sx = __fsub_rn(ox, a.x), sy = __fsub_rn(oy, a.y), sz = __fsub_rn(oz, a.z);
  const float u = __fmul_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(px, sx), __fmul_rn(py, sy)), __fmul_rn(pz, sz)), 0.0f), inv_det);
  if (u < 0.0f || u > 1.0f) return false;
  const float qx = __fsub_rn(__fmul_rn(sy, b.z), __fmul_rn(sz, b.y));
  const float qy = __fsub_rn(__fmul_rn(sz, b.x), __fmul_rn(sx, b.z));
  const float qz = __fsub_rn(__fmul_rn(sx, b.y), __fmul_rn(sy, b.x));
  const float v = __fmul_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(qx, dx), __fmul_rn(qy, dy)), __fmul_rn(qz, dz)), 0.0f), inv_det);
  if (v < 0.0f || __fadd_rn(u, v) > 1.0f) return false;
  const float t = __fmul_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(c.x, qx), __fmul_rn(c.y, qy)), __fmul_rn(c.z, qz)), 0.0f), inv_det);
  out.t = t; out.u = u; out.v = v;
  const bool outside = (u < 0.0f) | (u > 1.0f) | (v < 0.0f) | (__fadd_rn(u, v) > 1.0f);
  return !outside & (t > 0.0f) & ((t < best) | ((t == best) & (__float_as_int(b.w) < best_rank)));
}

// Cull factor for the distance test: a child is skipped when its entry distance exceeds
// the best t by more than 2^-10 relative.
__device__ __forceinline__ float cull_bound(float best) { return best * 1.0009765625f; }
// the smallest float above cull_bound(best) (best > 0), +inf when the bound is +inf
__device__ __forceinline__ float cull_up(float best) {
  const float cb = cull_bound(best);
  return isinf(cb) ? cb : __int_as_float(__float_as_int(cb) + 1);
}

// ---- resumable walk for the persistent kernels ----
// The state of one ray's walk, so a warp can run its lanes' walks step by step and hand
// a lane a new ray as soon as its walk ends (the replenishing persistent warps of Aila
// and Laine, "Understanding the Efficiency of Ray Traversal on GPUs", HPG 2009). A walk
// holds at most two pending subtrees beside its stack: `link`, the next one, and `leaf`,
// a leaf met on the way whose triangles are still to be tested.
struct Walk {
  const float4* nodes;   // the scene of this ray (lanes of one warp may walk different scenes)
  const float4* tris;
  float dx, dy, dz;
  float ox_, oy_, oz_, ix_, iy_, iz_;   // origin and 1/direction
  __device__ __forceinline__ float ox() const { return ox_; }
  __device__ __forceinline__ float oy() const { return oy_; }
  __device__ __forceinline__ float oz() const { return oz_; }
  __device__ __forceinline__ float ix() const { return ix_; }
  __device__ __forceinline__ float iy() const { return iy_; }
  __device__ __forceinline__ float iz() const { return iz_; }
  // each component twice, the operand of the packed box tests (built where it is used:
  // a register pair per component would hold six more registers through the walk)
  __device__ __forceinline__ f32x2 ox2() const { return pk2(ox_, ox_); }
  __device__ __forceinline__ f32x2 oy2() const { return pk2(oy_, oy_); }
  __device__ __forceinline__ f32x2 oz2() const { return pk2(oz_, oz_); }
  __device__ __forceinline__ f32x2 ix2() const { return pk2(ix_, ix_); }
  __device__ __forceinline__ f32x2 iy2() const { return pk2(iy_, iy_); }
  __device__ __forceinline__ f32x2 iz2() const { return pk2(iz_, iz_); }
  float best, bu, bv;
  float best_up;         // cull_up(best)
  int best_tri, best_rank;
  int link, sp;          // LINK_NONE: nothing left to open, LINK_POP: the stack's next; a leaf link waits for `leaf`
  float link_t;          // entry distance of the subtree `link` (checked again when a hit shortens the ray)
  int leaf;              // (stream slot << 4) | triangles left of the pending leaf; 0 in the low bits: none
  bool exact;
};

__device__ __forceinline__ void walk_begin(const DevScene& sc, const RayIn& r, Walk& w) {
  w.nodes = sc.nodes;
  w.tris = sc.tris;

  w.dx = r.dx; w.dy = r.dy; w.dz = r.dz;
  const float ix = __frcp_rn(r.dx), iy = __frcp_rn(r.dy), iz = __frcp_rn(r.dz);
  w.exact = isinf(ix) || isinf(iy) || isinf(iz);
  w.ox_ = r.ox; w.oy_ = r.oy; w.oz_ = r.oz;
  w.ix_ = ix; w.iy_ = iy; w.iz_ = iz;
  w.best = r.tmax; w.bu = 0.0f; w.bv = 0.0f;
  w.best_up = cull_up(r.tmax);
  w.best_tri = -1; w.best_rank = -1;
  w.sp = 0;
  w.leaf = 0;
  w.link = sc.root_link;
  w.link_t = -__int_as_float(0x7f800000);
  if (w.link != LINK_NONE && sc.root_test) {
    float te;
    const bool h = w.exact ? box_ref(w.ox(), w.oy(), w.oz(), w.ix(), w.iy(), w.iz(), sc.root_lo.x, sc.root_hi.x, sc.root_lo.y,
                                     sc.root_hi.y, sc.root_lo.z, sc.root_hi.z, te)
                           : box_fast(w.ox(), w.oy(), w.oz(), w.ix(), w.iy(), w.iz(), sc.root_lo.x, sc.root_hi.x, sc.root_lo.y,
                                      sc.root_hi.y, sc.root_lo.z, sc.root_hi.z, __int_as_float(0x7f800000), false, te);
    if (!h) w.link = LINK_NONE;
  }
  if (w.link < 0) {   // the whole scene is one leaf
    w.leaf = ~w.link;
    w.link = LINK_NONE;
  }
}

// A walk's stack of (subtree link, entry distance) pairs, at most `cap` deep: entries
// [0, n_smem) in this thread's column of the block's shared memory (stride: the block
// size), deeper ones in its column of a global spill area (stride: the grid's threads),
// each entry one 64-bit word.
// A short shared part leaves more of the SM's unified L1 and shared memory to the node
// and triangle fetches; n_smem == cap (g unused) keeps the whole stack in shared memory.
struct WalkStack {
  int2* s;
  int2* g;
  int stride, gstride, n_smem, cap;
  __device__ __forceinline__ void put(int i, int link, float t) const {
    const int2 e = make_int2(link, __float_as_int(t));
    if (i < n_smem) s[i * stride] = e;
    else g[(size_t)(i - n_smem) * gstride] = e;
  }
  __device__ __forceinline__ int2 at(int i) const {
    return i < n_smem ? s[i * stride] : g[(size_t)(i - n_smem) * gstride];
  }
};

// A stack of links alone, in shared memory, for walks that look at no entry distance again: half the
// bytes, and a bank a lane where the links of (link, distance) pairs share 16 banks between 32 lanes (a
// million any-hit rays through 1,000 triangles 148 -> 146 us, through 30,000 265 -> 254).
struct LinkStack {
  int* s;
  int stride, cap;
  __device__ __forceinline__ void put(int i, int link, float) const { s[i * stride] = link; }
  __device__ __forceinline__ int at(int i) const { return s[i * stride]; }
};

// The link of a walk that has to take its next subtree from the stack. Popping is left to
// the next node step, so that a step has one place where lanes pop, together.
constexpr int LINK_POP = LINK_NONE - 1;
__device__ __forceinline__ int pop_link(const Walk& w) { return w.sp > 0 ? LINK_POP : LINK_NONE; }

// 32 bytes of a node (aligned to 32) in one load: lanes that walk different nodes read from
// different cache lines, and the L1 serves a line at a time however little of it a lane takes,
// so half as many loads are less of its time: a million incoherent rays through the glass sphere
// 447 -> 429 us, the traversal of a 1920x1080 pass over 260K triangles 3.13 -> 3.08 ms.
__device__ __forceinline__ void load32(const float4* p, ulonglong2& a, ulonglong2& b) {
  asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(a.x), "=l"(a.y), "=l"(b.x), "=l"(b.y) : "l"(p));
}

// One interior node of the two-child layout: returns the next node (the nearer child
// hit, the other one pushed), or pop_link when neither child is hit. LINK_NONE: nothing
// left to open (or the stack bound was reached).
template <class Stack>
__device__ __forceinline__ int visit2(Walk& w, bool any, int link, const Stack& st, WalkCount& wc,
                                      bool& overflow) {
  const float4* nd = w.nodes + 4 * (size_t)link;
  ulonglong2 nx, ny, nz, links;   // (lo pair, hi pair) of an axis
  load32(nd, nx, ny);
  load32(nd + 2, nz, links);
  const int2 n3 = make_int2((int)(unsigned)links.x, (int)(links.x >> 32));
  wc.nodes += 2;
  // (lo - o) * inv and (hi - o) * inv of both children, two packed operations per bound
  float ax0, ax1, bx0, bx1, ay0, ay1, by0, by1, az0, az1, bz0, bz1;
  up2(mul2(sub2(nx.x, w.ox2()), w.ix2()), ax0, ax1);
  up2(mul2(sub2(nx.y, w.ox2()), w.ix2()), bx0, bx1);
  up2(mul2(sub2(ny.x, w.oy2()), w.iy2()), ay0, ay1);
  up2(mul2(sub2(ny.y, w.oy2()), w.iy2()), by0, by1);
  up2(mul2(sub2(nz.x, w.oz2()), w.iz2()), az0, az1);
  up2(mul2(sub2(nz.y, w.oz2()), w.iz2()), bz0, bz1);
  float t0, t1;
  bool h0, h1;
  if (!w.exact) {   // hit and within the cull bound
    h0 = box_fast_ab(ax0, bx0, ay0, by0, az0, bz0, w.best_up, !any, t0);
    h1 = box_fast_ab(ax1, bx1, ay1, by1, az1, bz1, w.best_up, !any, t1);
  } else {
    h0 = box_ref_ab(ax0, bx0, ay0, by0, az0, bz0, t0);
    h1 = box_ref_ab(ax1, bx1, ay1, by1, az1, bz1, t1);
    const float cb = cull_bound(w.best);
    h0 = h0 && !(t0 > cb);
    h1 = h1 && !(t1 > cb);
  }
  h0 = h0 && n3.x != LINK_NONE;
  h1 = h1 && n3.y != LINK_NONE;
  if (!(h0 || h1)) return pop_link(w);
  const bool both = h0 && h1;
  const bool second = both ? t1 < t0 : h1;   // the child to open next
  if (both) {
    if (w.sp >= st.cap) { overflow = true; w.sp = 0; return LINK_NONE; }
    st.put(w.sp, second ? n3.x : n3.y, second ? t0 : t1);
    ++w.sp;
  }
  w.link_t = second ? t1 : t0;
  return second ? n3.y : n3.x;
}

// (t, link) compare-exchange: the smaller entry distance first
__device__ __forceinline__ void cx(float& ta, int& la, float& tb, int& lb) {
  if (tb < ta) {
    const float t = ta; ta = tb; tb = t;
    const int l = la; la = lb; lb = l;
  }
}

// One interior node of the four-child layout (yc_scene.h, wide nodes): the four child
// boxes are tested with the reference's slab arithmetic, two children per packed
// operation, the hits sorted by entry distance, the nearest returned and the others
// pushed farthest first (pushed in any order, the walk visited more nodes: 3.97 against
// 3.59 ms per 1080p pass of a 260K-triangle scene).
template <class Stack>
__device__ __forceinline__ int visit4(Walk& w, bool any, int link, const Stack& st, WalkCount& wc,
                                      bool& overflow) {
  const float INF = __int_as_float(0x7f800000);
  const float4* nd = w.nodes + 8 * (size_t)link;
  wc.nodes += 4;
  float t[4];
  int l[4];
  const int4 ln = __ldg(reinterpret_cast<const int4*>(nd + 6));
  l[0] = ln.x; l[1] = ln.y; l[2] = ln.z; l[3] = ln.w;
  float a[3][4], b[3][4];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ulonglong2 lo, hi;
    load32(nd + 2 * k, lo, hi);
    const f32x2 o = k == 0 ? w.ox2() : k == 1 ? w.oy2() : w.oz2();
    const f32x2 i = k == 0 ? w.ix2() : k == 1 ? w.iy2() : w.iz2();
    up2(mul2(sub2(lo.x, o), i), a[k][0], a[k][1]);
    up2(mul2(sub2(lo.y, o), i), a[k][2], a[k][3]);
    up2(mul2(sub2(hi.x, o), i), b[k][0], b[k][1]);
    up2(mul2(sub2(hi.y, o), i), b[k][2], b[k][3]);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float te;
    bool h;
    if (!w.exact) {
      h = box_fast_ab(a[0][c], b[0][c], a[1][c], b[1][c], a[2][c], b[2][c], w.best_up, !any, te);
    } else {
      h = box_ref_ab(a[0][c], b[0][c], a[1][c], b[1][c], a[2][c], b[2][c], te);
      h = h && !(te >= w.best_up);
    }
    h = h && l[c] != LINK_NONE;
    t[c] = h ? te : INF;
    l[c] = h ? l[c] : LINK_NONE;
  }
  cx(t[0], l[0], t[1], l[1]);
  cx(t[2], l[2], t[3], l[3]);
  cx(t[0], l[0], t[2], l[2]);
  cx(t[1], l[1], t[3], l[3]);
  cx(t[1], l[1], t[2], l[2]);
  if (l[0] == LINK_NONE) return pop_link(w);
  const int extra = (l[1] != LINK_NONE) + (l[2] != LINK_NONE) + (l[3] != LINK_NONE);
  if (w.sp + extra > st.cap) { overflow = true; w.sp = 0; return LINK_NONE; }
#pragma unroll
  for (int c = 3; c >= 1; --c) {
    if (l[c] != LINK_NONE) {
      st.put(w.sp, l[c], t[c]);
      ++w.sp;
    }
  }
  w.link_t = t[0];
  return l[0];
}

// ---- steps of a walk ----
// A walk is a sequence of two kinds of step, opening an interior node and testing a leaf's
// triangles, and any order of a ray's pending steps gives its result (above). A lane that
// meets a leaf keeps it aside and goes on opening nodes (the postponed leaves of Aila and
// Laine) until it meets a second one. The warp takes one kind of step at a time, for all
// lanes that can take it (walk_wants_node, walk_wants_tri): the kind more of them can. Left to
// themselves (nodes until every lane has a leaf, then leaves until every lane has none)
// the lanes of a warp ran 12.8 at a time in nodes and 7.3 in triangles on the glass sphere's
// path rays, 8.2 and 3.1 on incoherent ones; with the vote 17.5 and 16.5, 16.3 and 14.7. The
// vote is two ballots a step, which four-child nodes (half as many steps) pay for: a
// million incoherent rays through the glass sphere 588 -> 448 us.
__device__ __forceinline__ bool walk_wants_node(const Walk& w) { return w.link >= 0 && w.link != LINK_NONE; }
__device__ __forceinline__ bool walk_wants_tri(const Walk& w) { return (w.leaf & 15) != 0; }

// a leaf met while none is pending is kept aside
__device__ __forceinline__ void walk_keep_leaf(Walk& w) {
  if (w.link < 0 && (w.leaf & 15) == 0) {
    w.leaf = ~w.link;
    w.link = pop_link(w);
  }
}

// The next subtree from the stack where one is due, then one interior node
// (walk_wants_node). `any` selects the any-hit rule, `overflow` is set when the stack
// bound was reached (the walk then ends early).
template <bool WIDE>
__device__ __forceinline__ void walk_node_step(Walk& w, bool any, const WalkStack& st, WalkCount& wc, bool& overflow) {
  while (w.link == LINK_POP) {
    --w.sp;
    const int2 e = st.at(w.sp);
    const float te = __int_as_float(e.y);
    w.link_t = te;
    w.link = te >= w.best_up ? pop_link(w) : e.x;   // (beyond the cull bound: the next one)
    walk_keep_leaf(w);
  }
  if (walk_wants_node(w)) {
    w.link = WIDE ? visit4(w, any, w.link, st, wc, overflow) : visit2(w, any, w.link, st, wc, overflow);
    walk_keep_leaf(w);
  }
}

// the triangles of the pending leaf (walk_wants_tri); an any-hit walk ends at its first hit
__device__ __forceinline__ void walk_leaf(Walk& w, bool any, WalkCount& wc) {
  const float4* tp = w.tris + 3 * (size_t)(w.leaf >> 4);
  int left = w.leaf & 15;
  w.leaf = 0;
  do {
    const float4 a = __ldg(tp + 0);
    const float4 b = __ldg(tp + 1);
    const float4 c = __ldg(tp + 2);
    tp += 3;
    ++wc.tris;
    TriHit th;
    if (tri_test(w.ox(), w.oy(), w.oz(), w.dx, w.dy, w.dz, a, b, c, w.best, w.best_rank, th)) {
      w.best = th.t;
      w.bu = th.u;
      w.bv = th.v;
      w.best_tri = __float_as_int(a.w);
      w.best_rank = __float_as_int(b.w);
      if (any) {
        w.link = LINK_NONE;
        return;
      }
    }
  } while (--left);
  w.best_up = cull_up(w.best);
  // the pending subtree, unless a hit put it out of reach
  if (w.link < LINK_POP && w.link_t >= w.best_up) w.link = pop_link(w);
  walk_keep_leaf(w);
}

// One step for the lanes of a warp that can take the kind more of them wait for; `nodes`
// and `tris` are the warp's ballots of walk_wants_node and walk_wants_tri, at least one of
// them not empty.
template <bool WIDE>
__device__ __forceinline__ void warp_walk_step(Walk& w, bool any, const WalkStack& st, WalkCount& wc, bool& overflow,
                                               unsigned nodes, unsigned tris) {
  if (__popc(nodes) >= __popc(tris)) {
    if (walk_wants_node(w)) walk_node_step<WIDE>(w, any, st, wc, overflow);
  } else {
    if (walk_wants_tri(w)) walk_leaf(w, any, wc);
  }
}

// The while-while loop of Aila and Laine without a vote on the kind of step, for any-hit rays over
// two-child nodes: every lane opens nodes until each of them has a leaf, then tests its leaves'
// triangles; true when the walk has ended. Such a walk keeps its segment's length until it stops, so
// no entry distance is looked at again. When to stop opening is asked of the lanes that happen to
// be together in the loop, as one group that is formed and asked with nothing in between: each of
// its lanes reaches the question, and no result depends on which lanes they are. (All lanes of the
// warp going round together, or a mask handed from round to round, take 2-4% longer from 50,000
// rays; no question at all 3-5% in large scenes.) Any-hit queries use it where the votes cost more
// than the lanes they bring together (trace.cu).
__device__ __forceinline__ bool any_walk_step(Walk& w, const LinkStack& st, WalkCount& wc, bool& overflow) {
  const auto pop = [&] { return w.sp > 0 ? st.at(--w.sp) : LINK_NONE; };
  int link = w.link, leaf = w.leaf;
  w.leaf = 0;
  while (link >= 0 && link != LINK_NONE) {
    link = visit2(w, true, link, st, wc, overflow);
    if (link == LINK_POP) link = pop();
    if (link < 0 && leaf == 0) {
      leaf = ~link;
      link = pop();
    }
    if (!cooperative_groups::coalesced_threads().any(leaf == 0)) break;
  }
  while (leaf != 0) {
    const float4* tp = w.tris + 3 * (size_t)(leaf >> 4);
    int left = leaf & 15;
    do {
      const float4 a = __ldg(tp + 0), b = __ldg(tp + 1), c = __ldg(tp + 2);
      tp += 3;
      ++wc.tris;
      TriHit th;
      if (tri_test(w.ox(), w.oy(), w.oz(), w.dx, w.dy, w.dz, a, b, c, w.best, w.best_rank, th)) {
        w.best = th.t;
        w.bu = th.u;
        w.bv = th.v;
        w.best_tri = __float_as_int(a.w);
        return true;
      }
    } while (--left);
    leaf = 0;
    if (link < 0) {   // a second leaf met on the way
      leaf = ~link;
      link = pop();
    }
  }
  w.link = link;
  return link == LINK_NONE;
}

}  // namespace yc
