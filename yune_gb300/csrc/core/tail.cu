// tail.cu -- the end of a pass, when few paths are left.
//
// A pass's last rounds carry few paths (long glass and mirror paths survive Russian
// roulette), and a round of the wavefront then lasts as long as its slowest ray: the GPU
// waits on one latency-bound walk per round while almost all of it idles. Once the paths
// left fit in one resident launch, k_tail gives each of them a lane that runs the same
// steps in turn -- walk the pending ray, store the hit, advance the state machine
// (logic_path) -- until the path writes its pixel. A warp's lanes walk together, the kind of
// step more of them can take at a time, and run their state machines together once every
// lane's ray is answered: the state machine's time is that of its code, whose phases a warp
// runs one after another whatever the lanes in them (25-65 thousand cycles a step), so the
// fewer runs the better (run when half the lanes wait: 1.65 ms against 1.40 ms on the glass
// sphere). With each lane on its own the kernel ran 3.5 lanes per instruction: 1.74 ms
// there against 1.10 ms (one ray at a time), and for a 256x256 frame of the Cornell box 1.10
// against 0.57 ms, 0.44 ms with its rays sent together. What bounds it is the longest chain
// of rays in a warp (12-25), at 600-1600 cycles a step of a walk. Every path computes exactly
// what the round-by-round wavefront computes (same state, same operations), so the pass's
// result is unchanged; paths no longer wait for each other between rays.
// The kernel is launched after every round's logic kernel on that round's output
// queues: above the threshold it returns at once; at or below it, it finishes the pass
// and its last block to exit empties the queues, so the remaining round launches find
// nothing to do.
#include <cuda_runtime.h>

#include "yc_internal.h"
#include "yc_trace_loop.cuh"
#include "yc_udpt.cuh"

namespace yc {

constexpr int TAIL_TB = 128;
// far more rays than any path can take (max_depth 100000, three rays per bounce); a
// path that reaches it is left unfinished and counted in DevStats::stack_overflow
constexpr int TAIL_MAX_RAYS = 1 << 22;
// Where a path sends two rays at once (logic_path) idle lanes of its warp walk the second ones, at
// least HELP_AT at a time while others walk (1, 8, 16 and 32 measured alike): four 512x512 passes
// of the Cornell box 1.30 ms of tail with both rays walked by the path's own lane, 1.06 ms now.
constexpr int HELP_AT = 8;

// three blocks per SM: up to 170 registers a thread, which the kernel needs without spills
template <bool WIDE, bool TOGETHER, bool MULTI>
__global__ void __launch_bounds__(TAIL_TB, 3) k_tail(PassParams pp, PathState ps, const int* __restrict__ in_closest,
                                                  const int* __restrict__ in_wait, RoundCounters* rc_in,
                                                  int threshold, int stack_cap, DevStats* st, int n_smem, int* spill) {
  __shared__ unsigned long long s_cnt[14];
  __shared__ bool s_last;
  const int nc = rc_in->n_closest, n = nc + rc_in->n_wait;
  if (n == 0 || n > threshold) return;   // uniform over the grid
  if (threadIdx.x < 14) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const WalkStack stack = thread_stack(stack_cap, n_smem, spill);
  const int lane = threadIdx.x & 31;
  const int warps = (int)(gridDim.x * (TAIL_TB / 32));
  const int quota = min(32, (n + warps - 1) / warps);   // lanes of a warp that take paths
  // per warp and lane: the segments of the lane's path found occluded, and the lanes of the
  // paths in `pend` in order
  __shared__ int s_occluded[TAIL_TB], s_pending[TAIL_TB];
  int* occluded = s_occluded + (threadIdx.x & ~31);
  int* pending = s_pending + (threadIdx.x & ~31);
  occluded[lane] = 0;
  const unsigned below = (1u << lane) - 1;
  LogicCounts lc;
  WalkCount wc;              // the current ray's walk
  unsigned overflow = 0;
  Walk w;
  w.link = LINK_NONE;
  w.leaf = 0;
  int p = -1, rays = 0;      // this lane's path, and the rays it has sent
  int todo = 0;              // its rays that no lane walks yet (EMIT_CLOSEST, EMIT_SEG0, EMIT_SEG1)
  int owner = -1, wp = -1, ray = 0;   // the lane of the path whose ray this lane walks, the path, the ray
  unsigned pend = 0;         // the lanes with todo (warp-uniform)
  bool more = true;          // the queues may still hold paths (warp-uniform)
  const auto begin = [&](int from, int path, int which) {
    owner = from;
    wp = path;
    ray = which;
    const float4 o = which == EMIT_CLOSEST ? ps.ro[path] : ps.hp[path];
    const float4 d = which == EMIT_SEG0 ? ps.wi[path] : ps.rd[path];
    if (which == EMIT_CLOSEST)
      walk_begin(pp.sc, RayIn{o.x, o.y, o.z, o.w, d.x, d.y, d.z}, w);
    else
      walk_begin(pp.sc, RayIn{ym::add(o.x, ym::mul(d.x, EPS_F)), ym::add(o.y, ym::mul(d.y, EPS_F)),
                              ym::add(o.z, ym::mul(d.z, EPS_F)), d.w, d.x, d.y, d.z}, w);
  };
  for (;;) {
    const unsigned nodes = __ballot_sync(0xffffffffu, walk_wants_node(w));
    const unsigned tris = __ballot_sync(0xffffffffu, walk_wants_tri(w));
    const unsigned idle = ~(nodes | tris);
    // (idle lanes wait until enough of them can take a ray at once)
    if (idle != 0xffffffffu && (!TOGETHER || !pend || __popc(idle) < min(HELP_AT, __popc(pend)))) {
      bool of = false;
      warp_walk_step<WIDE>(w, ray != EMIT_CLOSEST, stack, wc, of, nodes, tris);
      if (of) ++overflow;
      continue;
    }
    if (owner >= 0 && ((idle >> lane) & 1u)) {   // this lane's ray is answered
      unsigned long long* t = s_cnt + (ray != EMIT_CLOSEST ? 9 : 6);
      atomicAdd(t, 1ull);
      atomicAdd(t + 1, (unsigned long long)wc.nodes);
      atomicAdd(t + 2, (unsigned long long)wc.tris);
      wc.nodes = 0; wc.tris = 0;
      if (ray == EMIT_CLOSEST) ps.hit[wp] = make_float4(w.best, w.bu, w.bv, __int_as_float(w.best_tri));
      else if (w.best_tri >= 0) atomicOr(&occluded[owner], ray / EMIT_SEG0);
      owner = -1;
    }
    if (TOGETHER && pend) {   // the r-th idle lane takes a ray of the r-th path that has one left
      const int r = __popc(idle & below), r_own = __popc(pend & below), k = min(__popc(idle), __popc(pend));
      if (todo) pending[r_own] = lane;
      __syncwarp();
      const bool take = ((idle >> lane) & 1u) && r < k;
      const int from = take ? pending[r] : lane;
      const int tp = __shfl_sync(0xffffffffu, p, from), tt = __shfl_sync(0xffffffffu, todo, from);
      if (take) begin(from, tp, tt & -tt);
      if (todo && r_own < k) todo &= todo - 1;
      pend = __ballot_sync(0xffffffffu, todo != 0);
      continue;
    }
    // every ray is answered
    __syncwarp();
    const unsigned have = __ballot_sync(0xffffffffu, p >= 0);
    if (p >= 0) {
      if (occluded[lane]) ps.misc[p].z |= occluded[lane] << RECORD_BIT;
      occluded[lane] = 0;
      todo = logic_path<TOGETHER>(pp, MULTI ? pass_reset(pp, ps, p) : pp.reset, ps, p, lc, have) & ~EMIT_WAIT;
      rays += __popc(todo);
      if (todo && rays >= TAIL_MAX_RAYS) { ++overflow; todo = 0; }
      else if (MULTI && !todo && has_next_pass(pp, ps, p)) {
        const int pass = ps.job[p].w + 1;
        ps.job[p].w = pass;
        start_udpt(pp, ps, p, p % pp.width, p / pp.width, pp.seeds[pass]);
        lc.rays++; lc.trav++; lc.prim++;
        todo = EMIT_CLOSEST;
        rays = 0;
      }
      if (!todo) p = -1;
    }
    if (more) {
      const bool want = p < 0 && lane < quota;
      const unsigned m = __ballot_sync(0xffffffffu, want);
      int base = 0;
      if (lane == 0 && m) base = atomicAdd(&rc_in->work_logic, __popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (m && base + __popc(m) >= n) more = false;
      const int e = base + __popc(m & below);
      if (want && e < n) {
        p = e < nc ? in_closest[e] : in_wait[e - nc];
        todo = (e < nc ? EMIT_CLOSEST : 0) | segments_of(ps.misc[p].z);
        rays = 0;
      }
    }
    if (p >= 0) {   // a path's first ray is walked by its own lane
      begin(lane, p, todo & -todo);
      todo &= todo - 1;
    }
    if (TOGETHER) pend = __ballot_sync(0xffffffffu, todo != 0);
    if (!more && __ballot_sync(0xffffffffu, p >= 0) == 0) break;
  }
  const unsigned long long v[6] = {lc.rays, lc.ext, lc.shadow, lc.mis, lc.trav, lc.samples};
#pragma unroll
  for (int q = 0; q < 6; ++q)
    if (v[q]) atomicAdd(&s_cnt[q], v[q]);
  if (overflow) atomicAdd(&s_cnt[12], (unsigned long long)overflow);
  if (lc.prim) atomicAdd(&s_cnt[13], (unsigned long long)lc.prim);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long* dst[14] = {&st->rays, &st->extension, &st->shadow, &st->mis, &st->traversed, &st->samples,
                                   &st->ext_rays, &st->ext_boxes, &st->ext_tris, &st->any_rays, &st->any_boxes,
                                   &st->any_tris, &st->stack_overflow, &st->primary};
    for (int q = 0; q < 14; ++q)
      if (s_cnt[q]) atomicAdd(dst[q], s_cnt[q]);
    if (s_cnt[12]) atomicAdd(&st->call_overflow, s_cnt[12]);
    // the last block to finish empties the queues (every block has read the counts)
    __threadfence();
    s_last = atomicAdd(&rc_in->tail_exits, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_last) {
    rc_in->n_closest = 0;
    rc_in->n_any = 0;
    rc_in->n_wait = 0;
    rc_in->tail_exits = 0;
  }
}

static size_t tail_smem(int n) { return (size_t)TAIL_TB * n * sizeof(int2); }
static int tail_entries(int depth, int n_smem) { return n_smem > 0 && n_smem < depth + 2 ? n_smem : depth + 2; }

template <class K>
static int tail_grid_of(K kernel, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, TAIL_TB, smem);
  return per_sm > 0 ? per_sm * sms : -1;
}

using TailKernel = void (*)(PassParams, PathState, const int*, const int*, RoundCounters*, int, int, DevStats*, int, int*);
template <bool WIDE>
static TailKernel tail_kernel_of(bool together, bool multi) {
  if (together) return multi ? k_tail<WIDE, true, true> : k_tail<WIDE, true, false>;
  return multi ? k_tail<WIDE, false, true> : k_tail<WIDE, false, false>;
}
static TailKernel tail_kernel(const PassParams& pp) {
  const bool together = rays_together(pp), multi = pp.n_pass > 1;
  return pp.sc.wide ? tail_kernel_of<true>(together, multi) : tail_kernel_of<false>(together, multi);
}

int tail_capacity(const PassParams& pp, int n_smem, int* grid_out) {
  const size_t smem = tail_smem(tail_entries(pp.sc.depth, n_smem));
  const int grid = tail_grid_of(tail_kernel(pp), smem);
  if (grid_out) *grid_out = grid;
  return grid > 0 ? grid * TAIL_TB : 0;
}

int launch_tail(const PassParams& pp, const PathState& ps, const int* in_closest, const int* in_wait,
                RoundCounters* rc_in, int threshold, DevStats* st, int grid, cudaStream_t s, int n_smem, int* spill) {
  const int cap = pp.sc.depth + 2;
  n_smem = tail_entries(pp.sc.depth, spill ? n_smem : 0);
  const size_t smem = tail_smem(n_smem);
  const TailKernel kernel = tail_kernel(pp);
  kernel<<<grid, TAIL_TB, smem, s>>>(pp, ps, in_closest, in_wait, rc_in, threshold, cap, st, n_smem, spill);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace yc
