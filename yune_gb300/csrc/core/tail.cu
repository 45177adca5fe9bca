// tail.cu -- the tail kernel of unidirectional passes (yc_tail.cuh).
#include <cuda_runtime.h>

#include "yc_tail.cuh"
#include "yc_udpt.cuh"

namespace yc {

template <bool TOGETHER, bool MULTI>
struct UdptStep {
  static constexpr bool FAN = TOGETHER, BDPT = false;
  const PassParams& pp;
  const PathState& ps;
  __device__ __forceinline__ int segments(int p) const { return segments_of(ps.misc[p].z); }
  __device__ __forceinline__ int operator()(int p, unsigned mask, LogicCounts& lc) const {
    const int sent = logic_path<TOGETHER>(pp, MULTI ? pass_reset(pp, ps, p) : pp.reset, ps, p, lc, mask);
    if (!MULTI || sent || !has_next_pass(pp, ps, p)) return sent;
    const int pass = ps.job[p].w + 1;
    ps.job[p].w = pass;
    start_udpt(pp, ps, p, p % pp.width, p / pp.width, pp.seeds[pass]);
    lc.rays++; lc.trav++; lc.prim++;
    return EMIT_CLOSEST | NEW_PASS;
  }
};

// three blocks per SM: up to 170 registers a thread, which the kernel needs without spills
template <bool WIDE, bool TOGETHER, bool MULTI>
__global__ void __launch_bounds__(TAIL_TB, 3) k_tail(PassParams pp, PathState ps, Segments sg,
                                                  const int* __restrict__ in_closest, const int* __restrict__ in_wait,
                                                  RoundCounters* rc_in, int threshold, int stack_cap, DevStats* st,
                                                  int n_smem, int* spill) {
  tail_loop<WIDE>(UdptStep<TOGETHER, MULTI>{pp, ps}, pp.sc, ps, sg, in_closest, in_wait, rc_in, threshold, stack_cap, st,
                  n_smem, spill);
}

using TailKernel = void (*)(PassParams, PathState, Segments, const int*, const int*, RoundCounters*, int, int, DevStats*,
                            int, int*);
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
  kernel<<<grid, TAIL_TB, smem, s>>>(pp, ps, record_segments(ps), in_closest, in_wait, rc_in, threshold, cap, st, n_smem,
                                          spill);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace yc
