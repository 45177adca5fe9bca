// udpt.cu -- wavefront form of the unidirectional path tracer (kernels/legacy/udpt.cl).
//
// The reference runs one work-item per pixel through `shading` (udpt.cl:433-533),
// calling traceRay 2-3 times per bounce. Here every path is a small state machine in
// HBM (PathState) and a pass is a sequence of rounds:
//   raygen (a)   -> primary rays into the closest-hit queue
//   trace        -> extend kernel (b) on the closest-hit queue, occlusion kernel on the
//                   any-hit queue (NEE shadow rays and MIS BRDF rays, (d))
//   logic        -> advances each path whose rays are answered until it needs new ones
//                   (shading (c), light sampling and MIS (d), Russian roulette), up to
//                   two at once (logic_path); the new rays are appended to the next
//                   round's queues with warp prefixes and one atomic per warp and queue
//                   (e), so finished paths drop out and the queues stay dense.
// A path that finishes writes its colour into the running-mean accumulator
// (udpt.cl:193-210). The random numbers of a path are drawn in the reference order,
// from the same per-pixel xorshift stream.
#include <cuda_runtime.h>

#include "yc_internal.h"
#include "yc_udpt.cuh"

namespace yc {
// The first pass: the n pixels of the tile in the frame, `row` a row of it, one thread each. Their
// number is known, so every thread knows its place in the queue: with an append a warp the kernel
// was bound by its 260,000 atomics to two cache lines (1920x1080: 0.216 ms, now 0.111).
__global__ void __launch_bounds__(256) k_raygen(PassParams pp, int n, int row, PathState ps, int* q_closest,
                                                RoundCounters* rc, DevStats* st) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const int px = i % row + pp.off_x, py = i / row + pp.off_y, pix = py * pp.width + px;
    start_udpt(pp, ps, pix, px, py, pp.rand_seed);
    if (pp.n_pass > 1) ps.job[pix].w = 0;
    q_closest[i] = pix;
  }
  if (i == 0) {
    rc->n_closest = n;
    atomicAdd(&st->primary, (unsigned long long)n);
    atomicAdd(&st->rays, (unsigned long long)n);
    atomicAdd(&st->traversed, (unsigned long long)n);
  }
}

// the next pass of the paths in pp.q_restart
__global__ void __launch_bounds__(256) k_raygen_next(PassParams pp, PathState ps, int* q_closest, RoundCounters* rc,
                                                     DevStats* st) {
  const int n = rc->n_restart, lane = threadIdx.x & 31;
  for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += gridDim.x * blockDim.x) {
    int at = 0;
    if (lane == 0) at = atomicAdd(&rc->n_closest, min(32, n - base));
    at = __shfl_sync(0xffffffffu, at, 0) + lane;
    if (base + lane < n) {
      const int p = pp.q_restart[base + lane], pass = ps.job[p].w + 1;
      ps.job[p].w = pass;
      start_udpt(pp, ps, p, p % pp.width, p / pp.width, pp.seeds[pass]);
      q_closest[at] = p;
    }
  }
  if (n > 0 && blockIdx.x == 0 && threadIdx.x == 0) {
    atomicAdd(&st->primary, (unsigned long long)n);
    atomicAdd(&st->rays, (unsigned long long)n);
    atomicAdd(&st->traversed, (unsigned long long)n);
  }
}

void launch_raygen(const PassParams& pp, const PathState& ps, int* q_closest, RoundCounters* rc, DevStats* st,
                   cudaStream_t s) {
  const int n = tile_pixels(pp);
  if (n > 0) k_raygen<<<(n + 255) / 256, 256, 0, s>>>(pp, n, tile_row(pp), ps, q_closest, rc, st);
}
void launch_raygen_next(const PassParams& pp, const PathState& ps, int* q_closest, RoundCounters* rc, DevStats* st,
                        int grid, cudaStream_t s) {
  k_raygen_next<<<grid, 256, 0, s>>>(pp, ps, q_closest, rc, st);
}

// Two blocks per SM: with 129 registers or more, which the compiler otherwise takes for some forms of
// the step, one block is left and the shading takes 1.4 times as long.
template <bool TOGETHER, bool MULTI>
__global__ void __launch_bounds__(LOGIC_TB, 2) k_logic(PassParams pp, PathState ps, const int* __restrict__ in_closest,
                                                    const int* __restrict__ in_wait, const RoundCounters* rc_in,
                                                    int* out_closest, int* out_wait, int* q_any,
                                                    RoundCounters* rc_out,
                                                    DevStats* st, const int* __restrict__ sorted,
                                                    const SortCtl* sctl) {
  __shared__ unsigned long long s_cnt[8];   // rays, extension, shadow, mis, traversed, samples
  if (threadIdx.x < 8) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int nc = rc_in->n_closest, na = rc_in->n_wait;
  const int n = nc + na;
  const int lane = threadIdx.x & 31;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps_total = (gridDim.x * blockDim.x) >> 5;
  const bool use_sorted = sctl && sctl->use;
  for (int wbase = warp_global * 32; wbase < n; wbase += warps_total * 32) {
    const int e = wbase + lane;
    int emit = 0;
    int p = -1;
    LogicCounts lc;
    const unsigned mask = __ballot_sync(0xffffffffu, e < n);
    if (e < n) {
      p = use_sorted ? sorted[e] : (e < nc ? in_closest[e] : in_wait[e - nc]);
      emit = logic_path<TOGETHER>(pp, MULTI ? pass_reset(pp, ps, p) : pp.reset, ps, p, lc, mask);
    }
    RaysOut at;
    append_rays(emit, p, out_closest, out_wait, q_any, rc_out, at);
    if (MULTI) {   // paths that ended a pass and have another
      const bool again = e < n && !emit && has_next_pass(pp, ps, p);
      const unsigned m = __ballot_sync(0xffffffffu, again);
      int first = 0;
      if (lane == 0 && m) first = atomicAdd(&rc_out->n_restart, __popc(m));
      first = __shfl_sync(0xffffffffu, first, 0);
      if (again) pp.q_restart[first + __popc(m & ((1u << lane) - 1))] = p;
    }
    // counters
    unsigned v[6] = {lc.rays, lc.ext, lc.shadow, lc.conn, lc.trav, lc.samples};
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      unsigned x = v[q];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
      if (lane == 0 && x) atomicAdd(&s_cnt[q], (unsigned long long)x);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_cnt[0]) atomicAdd(&st->rays, s_cnt[0]);
    if (s_cnt[1]) atomicAdd(&st->extension, s_cnt[1]);
    if (s_cnt[2]) atomicAdd(&st->shadow, s_cnt[2]);
    if (s_cnt[3]) atomicAdd(&st->mis, s_cnt[3]);
    if (s_cnt[4]) atomicAdd(&st->traversed, s_cnt[4]);
    if (s_cnt[5]) atomicAdd(&st->samples, s_cnt[5]);
  }
}

void launch_logic(const PassParams& pp, const PathState& ps, const int* in_closest, const int* in_wait,
                  const RoundCounters* rc_in, int* out_closest, int* out_wait, int* q_any, RoundCounters* rc_out,
                  DevStats* st, int grid, cudaStream_t s, const int* sorted, const SortCtl* sctl) {
  const bool multi = pp.n_pass > 1;
  const auto kernel = rays_together(pp) ? (multi ? k_logic<true, true> : k_logic<true, false>)
                                        : (multi ? k_logic<false, true> : k_logic<false, false>);
  kernel<<<grid, LOGIC_TB, 0, s>>>(pp, ps, in_closest, in_wait, rc_in, out_closest, out_wait, q_any, rc_out, st, sorted,
                                    sctl);
}

// ---- tonemap (kernels/post-proc/tonemap.cl:14-47) ----
__global__ void k_tonemap(const float4* __restrict__ in, float4* __restrict__ out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 c = in[i];
  float y = ym::mul(0.212671f, c.x);
  y = ym::add(y, ym::mul(0.715160f, c.y));
  y = ym::add(y, ym::mul(0.072169f, c.z));
  y = ym::add(y, 0.001f);
  const float ldv = ym::div(ym::mul(y, ym::add(1.0f, ym::div(y, ym::mul(1.0f, 1.0f)))), ym::add(1.0f, y));
  const float g = ym::div(1.0f, 2.2f);
  float r[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) r[q] = ym::pow(ym::mul(ldv, ym::pow(ym::div(r[q], y), 1.0f)), g);
  out[i] = make_float4(r[0], r[1], r[2], r[3]);
}

void launch_tonemap(const float4* in, float4* out, int n, cudaStream_t s) {
  k_tonemap<<<(n + 255) / 256, 256, 0, s>>>(in, out, n);
}

}  // namespace yc
