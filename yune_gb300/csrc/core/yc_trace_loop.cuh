// yc_trace_loop.cuh -- the replenishing persistent traversal loop, shared by the per-pass
// trace kernels (trace.cu) and the batch engine (engine.cu).
#pragma once

#include "yc_internal.h"
#include "yc_shade.cuh"
#include "yc_traverse.cuh"

namespace yc {

constexpr int TRACE_TB = 128;       // block of the per-pass trace kernels
constexpr int TRACE_TB_MAX = 256;   // largest block of the batch engine's trace kernels

// warp-reduced traversal counters, one atomic per warp and counter
template <bool ANY>
__device__ __forceinline__ void flush_counts(DevStats* st, unsigned rays, const WalkCount& wc,
                                             unsigned long long overflow) {
  unsigned long long r = rays, nn = wc.nodes, tt = wc.tris;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    r += __shfl_xor_sync(0xffffffffu, r, off);
    nn += __shfl_xor_sync(0xffffffffu, nn, off);
    tt += __shfl_xor_sync(0xffffffffu, tt, off);
    overflow += __shfl_xor_sync(0xffffffffu, overflow, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (ANY) {
      if (r) atomicAdd(&st->any_rays, r);
      if (nn) atomicAdd(&st->any_boxes, nn);
      if (tt) atomicAdd(&st->any_tris, tt);
    } else {
      if (r) atomicAdd(&st->ext_rays, r);
      if (nn) atomicAdd(&st->ext_boxes, nn);
      if (tt) atomicAdd(&st->ext_tris, tt);
    }
    if (overflow) {
      atomicAdd(&st->stack_overflow, overflow);
      atomicAdd(&st->call_overflow, overflow);
    }
  }
}

// a path's closest-hit ray, and segment q
__device__ __forceinline__ RayIn path_ray(const SF<float4>& ro, const SF<float4>& rd, int p) {
  const float4 o = __ldg(&ro[p]), d = __ldg(&rd[p]);
  return RayIn{o.x, o.y, o.z, o.w, d.x, d.y, d.z};
}
__device__ __forceinline__ RayIn segment_ray(const Segments& sg, int q) {
  const float4 o = __ldg(&sg.org[sg.path(q)]), d = __ldg(sg.ray(q));
  return RayIn{ym::add(o.x, ym::mul(d.x, EPS_F)), ym::add(o.y, ym::mul(d.y, EPS_F)), ym::add(o.z, ym::mul(d.z, EPS_F)),
               d.w, d.x, d.y, d.z};
}

// Lanes refill when at least this many of a warp's 32 lanes are idle (a round's rays, whose
// neighbours walk alike, end closer together: 20 there measured 1% faster than 16, and 4%
// slower on incoherent ray queries).
constexpr int REFILL_AT = 16;
constexpr int REFILL_ROUND_AT = 20;

// The walk stack of this thread: its first n_smem entries in a column of the block's
// dynamic shared memory (stride: the block size), the rest of stack_cap in a column of
// `spill` (stride: the grid's threads; unused when n_smem == stack_cap)
__device__ __forceinline__ WalkStack thread_stack(int stack_cap, int n_smem, int* spill) {
  extern __shared__ int2 smem[];
  WalkStack ws;
  ws.s = smem + threadIdx.x;
  ws.stride = (int)blockDim.x;
  ws.gstride = (int)(gridDim.x * blockDim.x);
  ws.g = spill ? reinterpret_cast<int2*>(spill) + (blockIdx.x * blockDim.x + threadIdx.x) : nullptr;
  ws.cap = stack_cap;
  ws.n_smem = n_smem < stack_cap ? n_smem : stack_cap;
  return ws;
}

// The persistent loop shared by the kernels. Src supplies ray e of the work list and the
// scene it walks (begin) and stores its result (end). Each thread's stack is thread_stack.
// LANE (any-hit rays, two-child nodes): every lane takes its own steps (any_walk_step) instead of
// voted ones.
template <bool ANY, bool WIDE, bool LANE, class Src>
__device__ __forceinline__ void trace_loop(Src& src, int n, int* work, int stack_cap, DevStats* st,
                                           int n_smem = 1 << 30, int* spill = nullptr) {
  static_assert((ANY && !WIDE) || !LANE, "lane steps are for any-hit rays over two-child nodes");
  const WalkStack stack = thread_stack(stack_cap, n_smem, spill);
  const LinkStack links{reinterpret_cast<int*>(stack.s - threadIdx.x) + threadIdx.x, stack.stride, stack_cap};   // (LANE)
  const int lane = threadIdx.x & 31;
  unsigned long long overflow = 0;
  WalkCount wc;
  unsigned rays = 0;
  Walk w;
  w.link = LINK_NONE;
  w.leaf = 0;
  int e_cur = -1;            // work-list entry of this lane's ray, -1 when it has none
  bool more = true;          // the work list may still hold rays (warp-uniform)
  // A list shorter than half the launch's lanes is spread over its warps, two of each
  // scheduler's four or five in work, so that a warp's lanes wait for as few other walks as
  // there need be (1,172 closest-hit rays through a 300K-triangle scene 147 -> 58 us, 20,000
  // 188 -> 114 us, index included).
  const int warps = (int)(gridDim.x * blockDim.x) >> 6;   // half of them
  // (Lane by lane only below half of that: 50,000 any-hit rays through 34 triangles 30.1 -> 27.6 us.)
  const int even = min(32, max(1, (n + warps - 1) / warps));
  const int quota = LANE && even > 16 ? 32 : even;
  const unsigned takers = 0xffffffffu >> (32 - quota);   // the lanes that take rays
  const int refill = quota < 32 ? (quota + 1) / 2 : REFILL_AT;
  auto finish = [&]() {   // hands over the result of this lane's ray
    HitOut h;
    h.t = w.best; h.u = w.bu; h.v = w.bv; h.tri = w.best_tri;
    src.end(e_cur, h);
    e_cur = -1;
  };
  for (;;) {
    unsigned nodes = 0, tris = 0, idle;
    if (LANE) {
      idle = ~__ballot_sync(0xffffffffu, e_cur >= 0);
    } else {
      nodes = __ballot_sync(0xffffffffu, walk_wants_node(w));
      tris = __ballot_sync(0xffffffffu, walk_wants_tri(w));
      idle = ~(nodes | tris);
    }
    const unsigned take = idle & takers;   // (some lane, in the branch: the cursor moves on)
    if (idle == 0xffffffffu || (more && __popc(take) >= refill)) {
      if (!LANE && ((idle >> lane) & 1u) && e_cur >= 0) finish();
      if (!more) break;   // only when every lane is idle
      int base = 0;
      if (lane == 0) base = atomicAdd(work, __popc(take));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + __popc(take) >= n) more = false;
      const int e = base + __popc(take & ((1u << lane) - 1));
      if (((take >> lane) & 1u) && e < n) {
        e_cur = e;
        RayIn r;
        const DevScene& sc = src.begin(e, r);
        walk_begin(sc, r, w);
        ++rays;
      }
      if (!LANE) continue;
    }
    bool of = false;
    if (LANE) {
      if (e_cur >= 0 && any_walk_step(w, links, wc, of)) finish();
    } else {
      warp_walk_step<WIDE>(w, ANY, stack, wc, of, nodes, tris);
    }
    if (of) ++overflow;
  }
  flush_counts<ANY>(st, rays, wc, overflow);
}

// The same loop over both queues of a round in one launch: entries [0, nc) are the
// closest-hit rays, [nc, n) the any-hit rays (Src::begin and Src::end take the entry and
// its kind). One launch over all of a round's rays keeps its warps refilling for longer
// than two launches over half of them each: the lanes a warp leaves idle once the work
// list runs dry are a smaller share of the launch. Each lane counts its walk's work
// under its ray's kind.
// The per-kind totals (rays, child boxes and triangles of closest-hit and any-hit walks)
// are kept in shared memory, added once per finished ray, rather than in six registers
// of every thread for the whole launch.
template <bool WIDE, class Src>
__device__ __forceinline__ void trace_loop_mixed(Src& src, int nc, int n, int* work, int stack_cap, DevStats* st,
                                                 int n_smem = 1 << 30, int* spill = nullptr) {
  __shared__ unsigned s_tot[6];   // closest: rays, boxes, triangles; any-hit: the same
  if (threadIdx.x < 6) s_tot[threadIdx.x] = 0;
  __syncthreads();
  const WalkStack stack = thread_stack(stack_cap, n_smem, spill);
  const int lane = threadIdx.x & 31;
  unsigned overflow = 0;
  WalkCount wc;   // the current ray's walk
  Walk w;
  w.link = LINK_NONE;
  w.leaf = 0;
  int e_cur = -1;
  bool any = false;
  bool more = true;
  for (;;) {
    const unsigned nodes = __ballot_sync(0xffffffffu, walk_wants_node(w));
    const unsigned tris = __ballot_sync(0xffffffffu, walk_wants_tri(w));
    const unsigned idle = ~(nodes | tris);
    if (idle == 0xffffffffu || (more && __popc(idle) >= REFILL_ROUND_AT)) {
      const bool mine = (idle >> lane) & 1u;
      if (mine && e_cur >= 0) {
        HitOut h;
        h.t = w.best; h.u = w.bu; h.v = w.bv; h.tri = w.best_tri;
        src.end(e_cur, any, h);
        unsigned* t = s_tot + (any ? 3 : 0);
        atomicAdd(t, 1u);
        atomicAdd(t + 1, wc.nodes);
        atomicAdd(t + 2, wc.tris);
        wc.nodes = 0; wc.tris = 0;
        e_cur = -1;
      }
      if (!more) break;   // only when every lane is idle
      int base = 0;
      if (lane == 0) base = atomicAdd(work, __popc(idle));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + __popc(idle) >= n) more = false;
      const int e = base + __popc(idle & ((1u << lane) - 1));
      if (mine && e < n) {
        e_cur = e;
        any = e >= nc;
        RayIn r;
        const DevScene& sc = src.begin(e, any, r);
        walk_begin(sc, r, w);
      }
      continue;
    }
    bool of = false;
    warp_walk_step<WIDE>(w, any, stack, wc, of, nodes, tris);
    if (of) ++overflow;
  }
  unsigned long long of = overflow;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) of += __shfl_xor_sync(0xffffffffu, of, off);
  if (lane == 0 && of) {
    atomicAdd(&st->stack_overflow, of);
    atomicAdd(&st->call_overflow, of);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long* dst[6] = {&st->ext_rays, &st->ext_boxes, &st->ext_tris, &st->any_rays, &st->any_boxes,
                                  &st->any_tris};
    for (int k = 0; k < 6; ++k)
      if (s_tot[k]) atomicAdd(dst[k], (unsigned long long)s_tot[k]);
  }
}

}  // namespace yc
