// noalloc.cu -- render pass over one image tile that allocates nothing.
//
// Some callers cannot allocate device memory at the time they render: a real-time loop
// where cudaMalloc's implicit device synchronisation would stall the frame, or a host
// whose device memory belongs to its own allocator and forbids driver allocations
// after start-up. yc_render_pass sizes its wavefront state to the image on first use
// (cudaMalloc); this variant keeps that state -- the per-path records, the ray queues and
// the round counters -- in one file-scope __device__ array of NOALLOC_BYTES instead, so
// a tile of at most NOALLOC_MAX_PATHS pixels renders with no allocation at all. The
// array is part of the library image: every GPU that loads the library holds it until
// the process exits.
//
// Every call shares that one array, and it keeps the previous call's contents: the round
// counters are cleared on each pass, everything else is written before it is read. Two
// calls whose work overlaps on the GPU (two contexts on one device, on different
// streams) race on the array and must be serialised by the caller.
#include <cuda_runtime.h>

#include "yc_internal.h"
#include "yc_noalloc.h"
#include "yc_shade.cuh"

namespace yc {

// per-path bytes: the path record (PS_STRIDE float4, 224) + 4 queue slots + 2 segments (24)
constexpr size_t NOALLOC_PATH_BYTES = PS_STRIDE * 16 + 6 * 4;
constexpr size_t NOALLOC_BYTES = (size_t)NOALLOC_MAX_PATHS * NOALLOC_PATH_BYTES + 2 * sizeof(RoundCounters);

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];

namespace {

// Device address of the scratch array on the current device. In host code the array's
// name is only a host-side stand-in, so the address comes from cudaGetSymbolAddress. It
// is looked up on every call (a call already synchronises its stream, and the lookup is
// a table read): after a cudaDeviceReset or a new primary context the module is loaded
// again and the array may have moved, so no address is kept from an earlier call.
int scratch_address(unsigned char** out) {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return -1;
  *out = static_cast<unsigned char*>(p);
  return 0;
}

}  // namespace

// pathtracer prologue + createRay (kernels/legacy/udpt.cl:158-189, 213-238) for one
// tile; the path slot is the pixel's index inside the tile, so the state fits the
// tile-sized scratch.
__global__ void __launch_bounds__(256) k_raygen_tile(PassParams pp, int n, int row, PathState ps, int* q_closest,
                                                     RoundCounters* rc, DevStats* st) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = gid < n;
  const int px = gid % row + pp.off_x, py = gid / row + pp.off_y;
  const int pix = py * pp.width + px;
  if (active) {
    uint32_t seed;
    const f4 d = camera_direction(pp, px, py, pp.rand_seed, seed);
    const f4 o = ym::mk(pp.cam.r1.w, pp.cam.r2.w, pp.cam.r3.w, pp.cam.r4.w);
    float len = __int_as_float(0x7f800000);
    int k = -1;
    light_test(pp.sc, o, d, len, k);
    ps.misc[gid] = make_int4((int)seed, pix, 0 | ((k + 1) << 20), 0);   // state S_PRIMARY, no flags, no light j
    ps.ro[gid] = make_float4(o.x, o.y, o.z, len);
    ps.rd[gid] = make_float4(d.x, d.y, d.z, d.w);
  }
  if (active) q_closest[gid] = gid;
  if (gid == 0) {
    rc->n_closest = n;
    atomicAdd(&st->primary, (unsigned long long)n);
    atomicAdd(&st->rays, (unsigned long long)n);
    atomicAdd(&st->traversed, (unsigned long long)n);
  }
}

int noalloc_render(const NoallocPass& a, std::string& err) {
  const int n_paths = a.pp.tile_w * a.pp.tile_h;
  if (n_paths > NOALLOC_MAX_PATHS) {
    err = "tile of " + std::to_string(n_paths) + " pixels exceeds the " + std::to_string(NOALLOC_MAX_PATHS) +
          "-pixel scratch of yc_render_pass_noalloc; split the frame with block_x/block_y";
    return YC_E_INVALID;
  }
  unsigned char* base = nullptr;
  if (scratch_address(&base)) {
    err = "cudaGetSymbolAddress failed for the render scratch";
    return YC_E_LAUNCH;
  }
  // carve the scratch: the path records, 4 queues, the segments' queue, 2 round-counter blocks
  const size_t N = NOALLOC_MAX_PATHS;
  float4* f = reinterpret_cast<float4*>(base);
  const PathState ps = path_state_at(f);
  int* q = reinterpret_cast<int*>(f + PS_STRIDE * N);
  int* qs[4] = {q, q + N, q + 2 * N, q + 3 * N};
  int* q_any = q + 4 * N;
  RoundCounters* rc = reinterpret_cast<RoundCounters*>(q + 6 * N);
  const Segments sg = record_segments(ps);
  cudaStream_t s = a.stream;
  auto launch_failed = [&](const char* what) {
    const cudaError_t e = cudaPeekAtLastError();
    if (e == cudaSuccess) return false;
    err = std::string(what) + ": " + cudaGetErrorString(e);
    return true;
  };
  // the counters keep the previous call's values: clear both blocks first
  if (cudaMemsetAsync(rc, 0, 2 * sizeof(RoundCounters), s) != cudaSuccess) {
    err = "clearing the round counters failed";
    return YC_E_LAUNCH;
  }
  if (const int n = tile_pixels(a.pp))
    k_raygen_tile<<<(n + 255) / 256, 256, 0, s>>>(a.pp, n, tile_row(a.pp), ps, qs[0], rc, a.stats);
  if (launch_failed("ray generation")) return YC_E_LAUNCH;
  const int grid_c = trace_grid_blocks(false, a.pp.sc.depth, a.pp.sc.wide != 0);
  const int grid_a = trace_grid_blocks(true, a.pp.sc.depth, a.pp.sc.wide != 0);
  if (grid_c <= 0 || grid_a <= 0) {
    err = "trace kernel cannot be resident (stack too deep)";
    return YC_E_LAUNCH;
  }
  int cur = 0;
  bool finished = false;
  for (int round = 0; round < a.max_rounds; ++round) {
    RoundCounters* rin = rc + cur;
    RoundCounters* rout = rc + (1 - cur);
    if (launch_trace(a.pp.sc, qs[2 * cur], rin, ps, a.stats, grid_c, s) ||
        launch_trace_segments(a.pp.sc, q_any, rin, sg, a.stats, grid_a, s)) {
      launch_failed("trace kernel");
      if (err.empty()) err = "trace kernel launch failed";
      return YC_E_LAUNCH;
    }
    if (cudaMemsetAsync(rout, 0, sizeof(RoundCounters), s) != cudaSuccess) {
      err = "clearing the round counters failed";
      return YC_E_LAUNCH;
    }
    launch_logic(a.pp, ps, qs[2 * cur], qs[2 * cur + 1], rin, qs[2 * (1 - cur)], qs[2 * (1 - cur) + 1], q_any, rout,
                 a.stats, a.logic_grid, s);
    if (launch_failed("shading kernel")) return YC_E_LAUNCH;
    cur = 1 - cur;
    if ((round + 1) % 6 == 0 || round + 1 == a.max_rounds) {
      if (cudaMemcpyAsync(a.rc_host, rc + cur, sizeof(RoundCounters), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
          cudaStreamSynchronize(s) != cudaSuccess) {
        launch_failed("render pass");
        if (err.empty()) err = "render pass failed";
        return YC_E_LAUNCH;
      }
      if (a.rc_host->n_closest == 0 && a.rc_host->n_any == 0) { finished = true; break; }
    }
  }
  if (!finished) {
    err = "pass not finished after " + std::to_string(a.max_rounds) + " rounds (YC_OPT_MAX_ROUNDS)";
    return YC_E_TIMEOUT;
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("render pass failed: ") + cudaGetErrorString(e);
    return YC_E_LAUNCH;
  }
  return YC_OK;
}

}  // namespace yc
