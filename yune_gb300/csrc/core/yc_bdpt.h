// yc_bdpt.h -- buffers and launchers of the BDPT wavefront (bdpt.cu).
#pragma once

#include <cuda_runtime.h>

#include "yc_internal.h"
#include "../ym_math.h"

namespace yc {

// states of a BDPT path (misc.z & 15)
enum : int {
  // states that wait for a trace result
  B_LIGHT = 0,   // closest hit of the light-subpath ray that makes light vertex i
  B_EYE0 = 1,    // closest hit of the camera ray
  B_EYE = 2,     // closest hit of the eye-subpath ray that makes eye vertex i
  B_FAN = 3,     // segments from eye vertex i: to a light (next-event estimate) and to light vertices
  // transient phases
  Q_LIGHT_SAMPLE = 8,
  Q_EYE_START = 9,
  Q_EYE_SAMPLE = 10,
  Q_VERTEX = 11,
  Q_CONNECT = 12,
  Q_SEGMENTS = 13,
  Q_FINISH = 14
};

// subpath vertices, one 64-byte record (4 float4 fields) per vertex: vertex k of path p,
// field f at [(p * bounces + k) * 4 + f]; `bounces` vertices per subpath (BDPT_BOUNCES)
struct BdptBuffers {
  float4* lv;
  float4* ev;
  size_t N;
  int bounces;
  Segments sg;    // the segments of the round, at seg[(p << sg.shift) + s],
  float4* seg;
  int* q_any;     // and their queue
};

#ifdef __CUDACC__
// the segments a path collects in one step
struct FanOut {
  unsigned long long js = 0;   // which light vertex each goes to, a byte each (0: a light)
  int n = 0;
  __device__ __forceinline__ bool full(const BdptBuffers& bb) const { return n >> bb.sg.shift; }
  __device__ __forceinline__ void add(const BdptBuffers& bb, int p, int j, const ym::f4& dir, float len) {
    bb.seg[((size_t)p << bb.sg.shift) + n] = make_float4(dir.x, dir.y, dir.z, len);
    js |= (unsigned long long)j << (8 * n);
    ++n;
  }
};
// a path's traced segments: which are free, and the light vertex of each
struct FanIn {
  unsigned long long js;
  unsigned free;
  __device__ __forceinline__ void load(const int4& job, const int4& misc) {
    js = (unsigned)job.x | ((unsigned long long)(unsigned)job.y << 32);
    free = ~((unsigned)misc.z >> FAN_BIT) & ((1u << job.z) - 1u);
  }
  __device__ __forceinline__ int vertex(int s) const { return (int)(js >> (8 * s)) & 255; }
};

// the queue entries of a warp's lanes: paths with a closest-hit ray (emit 1), and paths that wait
// for `segs` segments (emit 2) with the segments themselves; all 32 lanes call it
__device__ __forceinline__ void append_bdpt(const BdptBuffers& bb, int emit, int p, int segs, int* out_closest,
                                            int* out_wait, RoundCounters* rc_out) {
  const int lane = threadIdx.x & 31;
  const unsigned mc = __ballot_sync(0xffffffffu, emit == 1), mf = __ballot_sync(0xffffffffu, emit == 2);
  const unsigned below = (1u << lane) - 1;
  int incl = emit == 2 ? segs : 0;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += u;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  int bc = 0, bf = 0, bs = 0;
  if (lane == 0) {
    if (mc) bc = atomicAdd(&rc_out->n_closest, __popc(mc));
    if (mf) bf = atomicAdd(&rc_out->n_wait, __popc(mf));
    if (total) bs = atomicAdd(&rc_out->n_any, total);
  }
  bc = __shfl_sync(0xffffffffu, bc, 0);
  bf = __shfl_sync(0xffffffffu, bf, 0);
  bs = __shfl_sync(0xffffffffu, bs, 0);
  if (emit == 1) out_closest[bc + __popc(mc & below)] = p;
  if (emit == 2) {
    out_wait[bf + __popc(mf & below)] = p;
    int* q = bb.q_any + (bs + incl - segs);
    for (int k = 0; k < segs; ++k) q[k] = (p << bb.sg.shift) + k;
  }
}
#endif

void launch_raygen_bdpt(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, int* q_closest,
                        RoundCounters* rc, DevStats* st, cudaStream_t s);
void launch_logic_bdpt(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                       const int* in_wait, const RoundCounters* rc_in, int* out_closest, int* out_wait,
                       RoundCounters* rc_out, DevStats* st, int grid, cudaStream_t s, const int* sorted = nullptr,
                       const SortCtl* sctl = nullptr);
// the bidirectional tracer with multiple importance sampling (bdpt_mis.cu): same buffers,
// same trace-state numbering (B_LIGHT .. B_FAN), light vertices only
void launch_raygen_bdpt_mis(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, int* q_closest,
                            RoundCounters* rc, DevStats* st, cudaStream_t s);
void launch_logic_bdpt_mis(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                           const int* in_wait, const RoundCounters* rc_in, int* out_closest, int* out_wait,
                           RoundCounters* rc_out, DevStats* st, int grid, cudaStream_t s, const int* sorted = nullptr,
                           const SortCtl* sctl = nullptr);

// tail kernels (yc_tail.cuh): blocks of one resident launch, and the launch
int tail_bdpt_grid(const PassParams& pp, int n_smem);
int tail_bdpt_mis_grid(const PassParams& pp, int n_smem);
int launch_tail_bdpt(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                     const int* in_wait, RoundCounters* rc_in, int threshold, DevStats* st, int grid, cudaStream_t s,
                     int n_smem, int* spill);
int launch_tail_bdpt_mis(const PassParams& pp, const PathState& ps, const BdptBuffers& bb, const int* in_closest,
                         const int* in_wait, RoundCounters* rc_in, int threshold, DevStats* st, int grid,
                         cudaStream_t s, int n_smem, int* spill);

}  // namespace yc
