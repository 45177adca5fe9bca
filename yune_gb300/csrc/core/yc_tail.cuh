// yc_tail.cuh -- the end of a pass, when few paths are left.
//
// A pass's last rounds carry few paths (long glass and mirror paths survive Russian
// roulette), and a round of the wavefront then lasts as long as its slowest ray: the GPU
// waits on one latency-bound walk per round while almost all of it idles. Once the paths
// left fit in one resident launch, the tail kernel gives each of them a lane that runs the same
// steps in turn -- walk the pending ray, store the hit, advance the state machine
// (Step) -- until the path writes its pixel. A warp's lanes walk together, the kind of
// step more of them can take at a time, and run their state machines together once every
// lane's ray is answered: the state machine's time is that of its code, whose phases a warp
// runs one after another whatever the lanes in them (34-48 thousand cycles a run in the
// mean), so the fewer runs the better (run when half the lanes wait: 1.65 ms against 1.40 ms on the glass
// sphere). With each lane on its own the kernel ran 3.5 lanes per instruction: 1.74 ms
// there against 1.10 ms (one ray at a time), and for a 256x256 frame of the Cornell box 1.10
// against 0.57 ms, 0.44 ms with its rays sent together. What bounds it is the longest chain of a
// warp: 13-17 runs, and the walks between them, at 1,800-2,900 cycles a step while its warps share
// their scheduler. (Counted with the clock on both sides of the two, in 256x256 and 256x192
// frames of the Cornell box and of 90K triangles; there the slowest warp takes two to three times
// the mean, half of it in the state machine in the box, three quarters in walks of 90K
// triangles.) Every path computes exactly what the round-by-round wavefront computes (same state,
// same operations), so the pass's result is unchanged; paths no longer wait for each other between
// rays.
// The kernel is launched after every round's logic kernel on that round's output
// queues: above the threshold it returns at once; at or below it, it finishes the pass
// and its last block to exit empties the queues, so the remaining round launches find
// nothing to do.
#pragma once

#include "yc_internal.h"
#include "yc_shade.cuh"
#include "yc_trace_loop.cuh"

namespace yc {

constexpr int TAIL_TB = 128;
// far more rays than any path can take (max_depth 100000, three rays per bounce); a
// path that reaches it is left unfinished and counted in DevStats::stack_overflow
constexpr int TAIL_MAX_RAYS = 1 << 22;
// Where a path sends two rays at once (logic_path) idle lanes of its warp walk the second ones, at
// least HELP_AT at a time while others walk (1, 8, 16 and 32 measured alike): four 512x512 passes
// of the Cornell box 1.30 ms of tail with both rays walked by the path's own lane, 1.06 ms now.
constexpr int HELP_AT = 8;

constexpr int NEW_PASS = 1 << 30;   // of a step's result: the path ended a pass and sends the first ray of its next

// step(p, mask, counts): one step of path p, by the lanes of `mask` together; the rays it sends
//   (EMIT_*), 0 when the path has ended
// step.segments(p): the segments in flight of a queued path
// Step::FAN: a path may send several rays at once; Step::BDPT: a bidirectional pass
template <bool WIDE, class Step>
__device__ __forceinline__ void tail_loop(const Step& step, const DevScene& sc, const PathState& ps, const Segments& sg,
                                          const int* __restrict__ in_closest, const int* __restrict__ in_wait,
                                          RoundCounters* rc_in, int threshold, int stack_cap, DevStats* st, int n_smem,
                                          int* spill) {
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
  int todo = 0;              // its rays that no lane walks yet (EMIT_CLOSEST, EMIT_SEG0 << s)
  int owner = -1, wp = -1, ray = 0;   // the lane of the path whose ray this lane walks, the path, the ray
  unsigned pend = 0;         // the lanes with todo (warp-uniform)
  bool more = true;          // the queues may still hold paths (warp-uniform)
  const auto begin = [&](int from, int path, int which) {
    owner = from;
    wp = path;
    ray = which;
    if (which == EMIT_CLOSEST) {
      const float4 o = ps.ro[path], d = ps.rd[path];
      walk_begin(sc, RayIn{o.x, o.y, o.z, o.w, d.x, d.y, d.z}, w);
    } else {
      const int s = __ffs(which) - 3;
      const float4 o = sg.org[path], d = *sg.ray((path << sg.shift) + s);
      walk_begin(sc, RayIn{ym::add(o.x, ym::mul(d.x, EPS_F)), ym::add(o.y, ym::mul(d.y, EPS_F)),
                           ym::add(o.z, ym::mul(d.z, EPS_F)), d.w, d.x, d.y, d.z}, w);
    }
  };
  for (;;) {
    const unsigned nodes = __ballot_sync(0xffffffffu, walk_wants_node(w));
    const unsigned tris = __ballot_sync(0xffffffffu, walk_wants_tri(w));
    const unsigned idle = ~(nodes | tris);
    // (idle lanes wait until enough of them can take a ray at once)
    if (idle != 0xffffffffu && (!Step::FAN || !pend || __popc(idle) < min(HELP_AT, __popc(pend)))) {
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
    if (Step::FAN && pend) {   // the r-th idle lane takes a ray of the r-th path that has one left
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
      if (occluded[lane]) ps.misc[p].z |= occluded[lane] << sg.bit;
      occluded[lane] = 0;
      todo = step(p, have, lc);
      rays = todo & NEW_PASS ? 1 : rays + __popc(todo);
      todo &= ~(EMIT_WAIT | NEW_PASS);
      if (todo && rays >= TAIL_MAX_RAYS) { ++overflow; todo = 0; }
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
        todo = (e < nc ? EMIT_CLOSEST : 0) | step.segments(p);
        rays = 0;
      }
    }
    if (p >= 0) {   // a path's first ray is walked by its own lane
      begin(lane, p, todo & -todo);
      todo &= todo - 1;
    }
    if (Step::FAN) pend = __ballot_sync(0xffffffffu, todo != 0);
    if (!more && __ballot_sync(0xffffffffu, p >= 0) == 0) break;
  }
  const unsigned long long v[6] = {lc.rays, lc.ext, lc.shadow, lc.conn, lc.trav, lc.samples};
#pragma unroll
  for (int q = 0; q < 6; ++q)
    if (v[q]) atomicAdd(&s_cnt[q], v[q]);
  if (overflow) atomicAdd(&s_cnt[12], (unsigned long long)overflow);
  if (lc.prim) atomicAdd(&s_cnt[13], (unsigned long long)lc.prim);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long* dst[14] = {&st->rays, &st->extension, &st->shadow, Step::BDPT ? &st->connection : &st->mis,
                                   &st->traversed, &st->samples, &st->ext_rays, &st->ext_boxes, &st->ext_tris,
                                   &st->any_rays, &st->any_boxes, &st->any_tris, &st->stack_overflow, &st->primary};
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

inline size_t tail_smem(int n) { return (size_t)TAIL_TB * n * sizeof(int2); }
inline int tail_entries(int depth, int n_smem) { return n_smem > 0 && n_smem < depth + 2 ? n_smem : depth + 2; }

// blocks of one resident launch
template <class K>
int tail_grid_of(K kernel, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, TAIL_TB, smem);
  return per_sm > 0 ? per_sm * sms : -1;
}

}  // namespace yc
