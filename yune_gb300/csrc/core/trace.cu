// trace.cu -- the extend (closest-hit) and occlusion (any-hit) kernels.
//
// Persistent kernels: one grid of (SM count x resident blocks) CTAs. A warp takes rays
// from a device cursor for its idle lanes (one atomic per refill) whenever at least
// REFILL_AT lanes are idle, and advances its busy lanes' walks by the kind of step more of
// them can take (yc_traverse.cuh), so lanes whose rays end early do not wait for the warp's
// longest ray. Each thread keeps its traversal stack in a column of dynamic shared
// memory (stride = block size, so the 32 lanes of a warp hit 32 different banks); the
// column holds depth + 1 entries of (link, entry distance). A walk that would overflow
// the stack is counted in DevStats::stack_overflow instead of writing out of bounds.
#include <cuda_runtime.h>

#include <algorithm>

#include "yc_internal.h"
#include "yc_shade.cuh"
#include "yc_trace_loop.cuh"

namespace yc {

// both queues of a round in one launch: closest-hit entries first, then the segments (or the
// sorted list, which keeps that split)
struct PathMixedSrc {
  const DevScene* sc;
  const int* __restrict__ q_closest;
  const int* __restrict__ q_any;
  const int* __restrict__ sorted;   // non-null: this round's sorted work list
  int nc;
  SF<float4> ro;
  SF<float4> rd;
  SF<float4> hit;
  Segments sg;
  __device__ __forceinline__ int entry(int e, bool any) const {
    return sorted ? sorted[e] : (any ? q_any[e - nc] : q_closest[e]);
  }
  __device__ __forceinline__ const DevScene& begin(int e, bool any, RayIn& r) {
    const int q = entry(e, any);
    r = any ? segment_ray(sg, q) : path_ray(ro, rd, q);
    return *sc;
  }
  __device__ __forceinline__ void end(int e, bool any, const HitOut& h) {
    const int q = entry(e, any);
    if (!any) hit[q] = make_float4(h.t, h.u, h.v, __int_as_float(h.tri));
    else if (h.tri >= 0) sg.occluded(q);
  }
};

template <bool WIDE>
__global__ void __launch_bounds__(TRACE_TB) k_trace_paths_mixed(DevScene sc, const int* __restrict__ q_closest,
                                                                const int* __restrict__ q_any, RoundCounters* rc,
                                                                SF<float4> ro, SF<float4> rd, SF<float4> hit,
                                                                Segments sg, int stack_cap, DevStats* st,
                                                                const int* sorted, const RaySortCtl* rs, int n_smem,
                                                                int* spill) {
  const int nc = rc->n_closest;
  PathMixedSrc src{&sc, q_closest, q_any, (rs && rs->use) ? sorted : nullptr, nc, ro, rd, hit, sg};
  trace_loop_mixed<WIDE>(src, nc, nc + rc->n_any, &rc->work_closest, stack_cap, st, n_smem, spill);
}

// one kind alone
template <bool ANY>
struct PathSrc {
  PathMixedSrc both;
  __device__ __forceinline__ const DevScene& begin(int e, RayIn& r) { return both.begin(e, ANY, r); }
  __device__ __forceinline__ void end(int e, const HitOut& h) { both.end(e, ANY, h); }
};

template <bool ANY, bool WIDE>
__global__ void __launch_bounds__(TRACE_TB) k_trace_paths(DevScene sc, const int* __restrict__ queue,
                                                          RoundCounters* rc, SF<float4> ro, SF<float4> rd,
                                                          SF<float4> hit, Segments sg, int stack_cap, DevStats* st) {
  PathSrc<ANY> src{{&sc, queue, queue, nullptr, 0, ro, rd, hit, sg}};
  trace_loop<ANY, WIDE, false>(src, ANY ? rc->n_any : rc->n_closest, ANY ? &rc->work_any : &rc->work_closest, stack_cap,
                               st);
}

// traceRay (udpt.cl:240-286) on explicit rays of 9 floats: light loop, then the BVH.
template <bool ANY>
struct RaySrc {
  const DevScene* sc;
  const float* __restrict__ rays;
  int* tri_out;
  float* t_out;
  int light;
  float len;
  __device__ __forceinline__ const DevScene& begin(int e, RayIn& r) {
    const float* q = rays + 9 * (size_t)e;
    const f4 o = ym::mk(q[0], q[1], q[2], q[3]);
    const f4 d = ym::mk(q[4], q[5], q[6], q[7]);
    len = q[8];
    light = -1;
    light_test(*sc, o, d, len, light);
    r = RayIn{o.x, o.y, o.z, len, d.x, d.y, d.z};
    return *sc;
  }
  __device__ __forceinline__ void end(int e, const HitOut& h) {
    if (ANY) {
      tri_out[e] = (h.tri >= 0 || light >= 0) ? 1 : 0;
      if (t_out) t_out[e] = h.tri >= 0 ? h.t : len;
    } else {
      tri_out[e] = h.tri;
      if (t_out) t_out[e] = h.tri >= 0 ? h.t : len;
      // a light hit is reported as -2 - light (unpacked by the host entry point)
      if (h.tri < 0 && light >= 0) tri_out[e] = -2 - light;
    }
  }
};

template <bool ANY, bool WIDE, bool LANE>
__global__ void __launch_bounds__(TRACE_TB) k_trace_rays(DevScene sc, const float* __restrict__ rays, int n,
                                                         int* work, int* tri_out, float* t_out, int stack_cap,
                                                         DevStats* st, int n_smem, int* spill) {
  RaySrc<ANY> src{&sc, rays, tri_out, t_out, -1, 0.0f};
  trace_loop<ANY, WIDE, LANE>(src, n, work, stack_cap, st, n_smem, spill);
}

static int stack_cap_for(int depth) { return depth + 2; }
static size_t smem_for(int cap) { return (size_t)TRACE_TB * 2 * cap * sizeof(int); }

static int g_sm_count = 0;

template <class K>
static int resident_grid(K kernel, size_t smem) {
  if (g_sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (g_sm_count <= 0) g_sm_count = 1;
  }
  int per_sm = 0;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, TRACE_TB, smem);
  if (per_sm <= 0) return -1;
  return g_sm_count * per_sm;
}

int trace_grid_blocks(bool any_hit, int depth, bool wide) {
  const size_t smem = smem_for(stack_cap_for(depth));
  if (wide) return any_hit ? resident_grid(k_trace_paths<true, true>, smem) : resident_grid(k_trace_paths<false, true>, smem);
  return any_hit ? resident_grid(k_trace_paths<true, false>, smem) : resident_grid(k_trace_paths<false, false>, smem);
}

template <bool ANY>
static int launch_alone(const DevScene& sc, const int* queue, RoundCounters* rc, SF<float4> ro, SF<float4> rd,
                        SF<float4> hit, const Segments& sg, DevStats* st, int grid_blocks, cudaStream_t s) {
  const int cap = stack_cap_for(sc.depth);
  const size_t smem = smem_for(cap);
  if (sc.wide) k_trace_paths<ANY, true><<<grid_blocks, TRACE_TB, smem, s>>>(sc, queue, rc, ro, rd, hit, sg, cap, st);
  else k_trace_paths<ANY, false><<<grid_blocks, TRACE_TB, smem, s>>>(sc, queue, rc, ro, rd, hit, sg, cap, st);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}
int launch_trace(const DevScene& sc, const int* queue, RoundCounters* rc, const PathState& ps, DevStats* st,
                 int grid_blocks, cudaStream_t s) {
  return launch_alone<false>(sc, queue, rc, ps.ro, ps.rd, ps.hit, Segments{}, st, grid_blocks, s);
}
int launch_trace_segments(const DevScene& sc, const int* q_any, RoundCounters* rc, const Segments& sg, DevStats* st,
                          int grid_blocks, cudaStream_t s) {
  return launch_alone<true>(sc, q_any, rc, {}, {}, {}, sg, st, grid_blocks, s);
}

static_assert(TRACE_TB == TRACE_TB_PASS, "the host sizes the per-pass spill area by TRACE_TB_PASS");
int trace_stack_cap(int depth) { return stack_cap_for(depth); }

int trace_mixed_grid_blocks(int depth, bool wide, int n_smem) {
  const int cap = stack_cap_for(depth);
  const size_t smem = smem_for(n_smem > 0 && n_smem < cap ? n_smem : cap);
  return wide ? resident_grid(k_trace_paths_mixed<true>, smem) : resident_grid(k_trace_paths_mixed<false>, smem);
}

int launch_trace_mixed(const DevScene& sc, const int* q_closest, const int* q_any, RoundCounters* rc,
                       const PathState& ps, const Segments& sg, DevStats* st, int grid_blocks, cudaStream_t s,
                       const int* sorted, const RaySortCtl* rs, int n_smem, int* spill) {
  const int cap = stack_cap_for(sc.depth);
  if (!(n_smem > 0 && n_smem < cap && spill)) n_smem = cap;
  const size_t smem = smem_for(n_smem);
  if (sc.wide)
    k_trace_paths_mixed<true><<<grid_blocks, TRACE_TB, smem, s>>>(sc, q_closest, q_any, rc, ps.ro, ps.rd, ps.hit, sg, cap,
                                                                  st, sorted, rs, n_smem, spill);
  else
    k_trace_paths_mixed<false><<<grid_blocks, TRACE_TB, smem, s>>>(sc, q_closest, q_any, rc, ps.ro, ps.rd, ps.hit, sg,
                                                                   cap, st, sorted, rs, n_smem, spill);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

// Any-hit queries over two-child nodes take their steps lane by lane, their stacks of links in shared
// memory, except the longest lists in large scenes, whose steps are voted. Lane by lane / voted, us:
//   triangles     4,096 rays   100,000     300,000     600,000       1M
//   34             19 / 20     33 / 34     53 / 58      87 / 99    135 / 161
//   1,000          32 / 38     46 / 52     66 / 75      99 / 112   148 / 170
//   10,000         44 / 53     77 / 87    116 / 119    179 / 183   266 / 264
//   30,000         43 / 54     86 / 93    114 / 125    171 / 187   256 / 273
//   81,954         62 / 74    111 / 122   163 / 163    226 / 219   325 / 315
//   300,000        71 / 90    132 / 148   180 / 186    273 / 276   383 / 382
// (Bound by lanes: 3-8 of 32 by lane, but with a third fewer instructions a step.)
constexpr int VOTE_SCENE = 1 << 16;    // triangles and
constexpr int VOTE_LIST = 1 << 19;     // segments from which the steps are voted
constexpr int LANE_STACK = 46;         // entries of a stack at most

static bool lane_steps(const DevScene& sc, bool any_hit, int n) {
  return any_hit && !sc.wide && stack_cap_for(sc.depth) <= LANE_STACK && (sc.n_tri < VOTE_SCENE || n < VOTE_LIST);
}
using RaysKernel = void (*)(DevScene, const float*, int, int*, int*, float*, int, DevStats*, int, int*);
static RaysKernel rays_kernel(const DevScene& sc, bool any_hit, int n) {
  if (!any_hit) return sc.wide ? k_trace_rays<false, true, false> : k_trace_rays<false, false, false>;
  if (sc.wide) return k_trace_rays<true, true, false>;
  return lane_steps(sc, any_hit, n) ? k_trace_rays<true, false, true> : k_trace_rays<true, false, false>;
}
static int rays_smem_entries(const DevScene& sc, int n_smem) {
  const int cap = stack_cap_for(sc.depth);
  return n_smem > 0 && n_smem < cap ? n_smem : cap;
}
// lane by lane the whole stack lies in shared memory, a link an entry
static size_t rays_smem(const DevScene& sc, bool any_hit, int n, int n_smem) {
  if (lane_steps(sc, any_hit, n)) return (size_t)TRACE_TB * stack_cap_for(sc.depth) * sizeof(int);
  return smem_for(rays_smem_entries(sc, n_smem));
}

int trace_rays_grid_blocks(const DevScene& sc, bool any_hit, int n, int n_smem) {
  const int grid = resident_grid(rays_kernel(sc, any_hit, n), rays_smem(sc, any_hit, n, n_smem));
  // (Lists that eight blocks per SM take at one ray a lane, and in scenes of short walks those of up
  // to three, are shared out better by eight than by nine. Eight / nine, us: 1,000 triangles, 100,000
  // rays 45.5 / 46.3, 300,000 66 / 67, 1M 150 / 147; 30,000 triangles, 150,000 rays 85 / 88, 200,000
  // 101 / 99, 600,000 176 / 171.)
  const bool short_list = n <= 8 * g_sm_count * TRACE_TB || (sc.n_tri < 4096 && n < 1 << 19);
  return lane_steps(sc, any_hit, n) && short_list && grid > 0 ? std::min(grid, 8 * g_sm_count) : grid;
}

int launch_trace_rays(const DevScene& sc, bool any_hit, const float* rays9, int n, int* tri_out, float* t_out,
                      int* work, DevStats* st, int grid, cudaStream_t s, int n_smem, int* spill) {
  n_smem = rays_smem_entries(sc, spill ? n_smem : 0);
  rays_kernel(sc, any_hit, n)<<<grid, TRACE_TB, rays_smem(sc, any_hit, n, n_smem), s>>>(
      sc, rays9, n, work, tri_out, t_out, stack_cap_for(sc.depth), st, n_smem, spill);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace yc
