// yc_internal.h -- host-side declarations shared by the core's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "yc_scene.h"
#include "yune_cuda.h"

namespace yc {

// ---- wavefront path state: one record of PS_STRIDE float4 (224 B, seven 32-byte
// sectors) per path slot ----
// The logic kernel reads and writes a path's whole record, and after the shade-queue
// sort neighbouring threads hold unrelated slots; one contiguous record per path keeps
// every sector it fetches fully used (a field per array would use half of each). The
// closest-hit ray shares a sector, so do the batch engine's (job, pass) pair and the hit, and
// a shadow ray's direction and origin.
// misc.x seed, misc.y pixel index, misc.z packed (state | flags << 4 | (j+1) << 12 |
// (k+1) << 20; the trace sets bit 28 when the path's shadow ray is occluded, bit 29 for its
// MIS ray), misc.w bounce index.
constexpr int PS_STRIDE = 14;
enum { PSF_RO = 0, PSF_RD, PSF_JOB, PSF_HIT, PSF_MISC, PSF_THR, PSF_THR_NEXT, PSF_DIRECT, PSF_INDIRECT, PSF_LS,
       PSF_HP, PSF_WI, PSF_WO, PSF_NRM };

// one field of every record: slot i at p[i * PS_STRIDE]
template <class T>
struct SF {
  T* p;
  __host__ __device__ __forceinline__ T& operator[](size_t i) const { return p[i * PS_STRIDE]; }
};

struct PathState {
  SF<int4> misc;
  SF<float4> thr;        // throughput
  SF<float4> thr_next;   // throughput after the pending bounce (udpt.cl:504-507)
  SF<float4> direct;     // direct_color (udpt.cl:455)
  SF<float4> indirect;   // indirect_color
  SF<float4> ls;         // light_sample of the NEE in flight (udpt.cl:562-563)
  SF<float4> hp;         // xyz hit point, w material index (int bits)
  SF<float4> nrm;        // xyz shading normal, w light_pdf
  SF<float4> wo;         // xyz w_o, w brdf_pdf of the MIS ray
  SF<float4> wi;         // the shadow ray: direction xyz, length
  SF<float4> ro;         // emitted closest-hit ray: origin xyz, length; or x brdf_prob of the MIS ray
  SF<float4> rd;         // emitted closest-hit ray: direction xyz; or the MIS ray: direction xyz, length
  SF<float4> hit;        // its result: (t, u, v, tri)
  SF<int4> job;          // batch engine: x, y = (job, pass) of the slot's pixel task; a call of several
                         // passes: w = the path's pass
};

// the path state of the records starting at rec (PS_STRIDE float4 per slot)
inline PathState path_state_at(float4* rec) {
  PathState ps;
  ps.misc = SF<int4>{reinterpret_cast<int4*>(rec + PSF_MISC)};
  ps.thr = SF<float4>{rec + PSF_THR};
  ps.thr_next = SF<float4>{rec + PSF_THR_NEXT};
  ps.direct = SF<float4>{rec + PSF_DIRECT};
  ps.indirect = SF<float4>{rec + PSF_INDIRECT};
  ps.ls = SF<float4>{rec + PSF_LS};
  ps.hp = SF<float4>{rec + PSF_HP};
  ps.nrm = SF<float4>{rec + PSF_NRM};
  ps.wo = SF<float4>{rec + PSF_WO};
  ps.wi = SF<float4>{rec + PSF_WI};
  ps.ro = SF<float4>{rec + PSF_RO};
  ps.rd = SF<float4>{rec + PSF_RD};
  ps.hit = SF<float4>{rec + PSF_HIT};
  ps.job = SF<int4>{reinterpret_cast<int4*>(rec + PSF_JOB)};
  return ps;
}

// Per-round device counters (cleared by one memset per round), each on a cache line of its own:
// every warp of the shading kernels appends to all three queues, and atomics to one line run
// one after another, about one a nanosecond (shading of four 512x512 passes of the Cornell box
// 1.83 ms with all in one line, 1.79 now).
struct RoundCounters {
  int n_closest;      // entries appended to the closest queue
  int pad0_[31];
  int n_any;          // entries appended to the any-hit queue
  int pad1_[31];
  int n_wait;         // paths without a closest-hit ray that wait for segments (n_any counts the segments)
  int pad2_[31];
  int work_closest;   // persistent-kernel work cursors
  int pad3_[31];
  int work_any;
  int pad4_[31];
  int work_logic;
  int tail_exits;     // blocks of the tail kernel that have left
  int pad5_[30];
  int n_restart;      // paths that ended a pass and have another
  int pad6_[31];
};

// The segments (any-hit rays) of a path: several may be in flight in one round, beside a
// closest-hit ray or instead of one. Segment s of path p is entry q = (p << shift) + s of the
// any-hit queue, its direction and length are at base[p * stride + s * step], its origin is
// org[p] moved along the direction by EPS_F, and a segment found occluded sets bit (bit + s) of
// misc[p].z, which the step that sends it writes.
// A path without a closest-hit ray that waits for segments is in the round's waiting queue.
//   unidirectional: the shadow and the MIS ray of a vertex, in the record (wi and rd, from hp)
//   bidirectional: the shadow rays of an eye vertex, to a light and to the light subpath's
//     vertices, up to 2^shift at once, in an array of their own (from ro); byte s of job.x,
//     job.y says which light vertex segment s goes to, job.z how many segments there are
struct Segments {
  const float4* base;
  SF<float4> org;
  SF<int4> misc;
  int stride, step, shift, bit;
#ifdef __CUDACC__
  __device__ __forceinline__ int path(int q) const { return q >> shift; }
  __device__ __forceinline__ int index(int q) const { return q & ((1 << shift) - 1); }
  __device__ __forceinline__ const float4* ray(int q) const {
    return base + ((long long)path(q) * stride + index(q) * step);
  }
  __device__ __forceinline__ void occluded(int q) const { atomicOr(&misc[path(q)].z, 1 << (bit + index(q))); }
#endif
};
constexpr int FAN_SHIFT = 3;
constexpr int FAN_BIT = 20, RECORD_BIT = 28;   // `bit` of the two
// the two segments of a unidirectional path
inline Segments record_segments(const PathState& ps) {
  return Segments{ps.wi.p, ps.hp, ps.misc, PS_STRIDE, PSF_RD - PSF_WI, 1, RECORD_BIT};
}

// Sorting of a round's traversal work list by ray origin and direction (raysort.cu):
// `use` tells the trace kernel whether this round's list is the sorted one.
struct RaySortCtl {
  int use;
  int pad[3];
};
#ifdef __CUDACC__
// ---- ray-sort key (raysort.cu, and the batch engine's producers) ----
__device__ __forceinline__ unsigned rs_spread3(unsigned x) {   // bit i of x -> bit 3i (x < 8)
  return (x & 1u) | ((x & 2u) << 2) | ((x & 4u) << 4);
}
__device__ __forceinline__ unsigned rs_cell_of(float v, float scale, int n) {
  const float c = fminf(fmaxf(v * scale, 0.0f), (float)(n - 1));   // NaN -> 0
  return (unsigned)(int)c;
}
// Morton code of the origin's cell in the scene box (ob bits per axis), then of the
// direction's cell in [-1, 1]^3 (db bits per axis)
__device__ __forceinline__ unsigned ray_key(const float4& o, const float4& d, const float4& lo, const float4& hi,
                                            int ob, int db) {
  const int no = 1 << ob, nd = 1 << db;
  const float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
  const unsigned ox = rs_cell_of(o.x - lo.x, ex > 0.0f ? (float)no / ex : 0.0f, no);
  const unsigned oy = rs_cell_of(o.y - lo.y, ey > 0.0f ? (float)no / ey : 0.0f, no);
  const unsigned oz = rs_cell_of(o.z - lo.z, ez > 0.0f ? (float)no / ez : 0.0f, no);
  const float hd = 0.5f * (float)nd;
  const unsigned dx = rs_cell_of(d.x + 1.0f, hd, nd), dy = rs_cell_of(d.y + 1.0f, hd, nd),
                 dz = rs_cell_of(d.z + 1.0f, hd, nd);
  const unsigned mo = rs_spread3(ox) | (rs_spread3(oy) << 1) | (rs_spread3(oz) << 2);
  const unsigned md = rs_spread3(dx) | (rs_spread3(dy) << 1) | (rs_spread3(dz) << 2);
  return (mo << (3 * db)) | md;
}
#endif

struct RaySortBufs {
  unsigned* keys;      // one per work-list entry (with keys_any: one per closest-hit queue entry)
  unsigned* keys_any;  // null, or the any-hit queue's keys (the batch engine's logic and fill
                       // kernels write both arrays and the histogram as they queue rays)
  unsigned* hist;      // raysort_bins(ob, db) counters, zero between rounds
  unsigned* cursor;    // scatter cursors (exclusive prefix of hist within its tile of 1024 bins)
  unsigned* blk_sum;   // tile totals (64 at most)
  int* sorted;         // the sorted work list (path indices)
  RaySortCtl* ctl;
  int ob, db;          // origin and direction bits per axis
  int jb;              // job bits of a batch's key (3 * (ob + db) + jb <= 15; 0 for one scene)
  int threshold;       // rounds with fewer rays are traced unsorted
};

// Sorting of the shade queue by the phase a path waits in (S_PRIMARY..S_EXT of the
// unidirectional path, B_LIGHT..B_CONN of BDPT) and material class (diffuse, glossy,
// mirror, dielectric, no surface): key = phase * 5 + class (engine.cu).
constexpr int SORT_KEYS = 25;
struct SortCtl {
  int use;                  // 1: this round's shade queue is the sorted one
  int pad_;
  int count[SORT_KEYS];     // paths per key
  int cursor[SORT_KEYS];    // scatter cursors (exclusive prefix of count)
};

// device-wide statistics (yc_stats layout, 64-bit counters); call_overflow counts the
// stack overflows of the current API call only (cleared when a call starts, read when it
// ends, so the call can return YC_E_OVERFLOW)
struct DevStats {
  unsigned long long rays, primary, extension, shadow, mis, connection, traversed, samples, stack_overflow;
  unsigned long long ext_rays, ext_boxes, ext_tris, any_rays, any_boxes, any_tris;
  unsigned long long call_overflow;
};

// the camera's aspect ratio as createRay computes it (udpt.cl:216-217, in double precision):
// one value per frame, computed on the host when a pass is set up
inline float frame_aspect(int width, int height) { return (float)(((double)width * 1.0) / (double)height); }

struct PassParams {
  DevScene sc;
  yc_cam cam;
  float4* accum;
  int width, height;
  double aspect;           // udpt.cl:216-217 in double precision, set by frame_aspect (a float value)
  double w, h, inv_w, inv_h;   // the frame's size and its reciprocals (frame_size)
  int tile_w, tile_h;      // work-item grid of one block launch
  int off_x, off_y;        // pixel offset of the block (udpt.cl:166-167)
  uint32_t rand_seed;      // of the first pass
  int reset;               // whether it starts the accumulator anew
  int gi_check;
  int mis, rr_threshold, max_depth, brdf_model, mis_lobe_fix;
  // several passes in one wavefront (n_pass > 1): their seeds, and the queue of paths to start again
  int n_pass;
  const uint32_t* seeds;
  int* q_restart;
};

// the pixels of the launch's tile that lie in the frame: a row of them, and their number
inline int tile_row(const PassParams& pp) {
  const int w = pp.width - pp.off_x;
  return w < pp.tile_w ? (w > 0 ? w : 0) : pp.tile_w;
}
inline int tile_pixels(const PassParams& pp) {
  const int h = pp.height - pp.off_y;
  return tile_row(pp) * (h < pp.tile_h ? (h > 0 ? h : 0) : pp.tile_h);
}

inline void frame_size(PassParams& pp, int width, int height) {
  pp.width = width;
  pp.height = height;
  pp.aspect = frame_aspect(width, height);
  pp.w = width;
  pp.h = height;
  pp.inv_w = 1.0 / pp.w;
  pp.inv_h = 1.0 / pp.h;
}

// refit.cu: the nodes of an uploaded scene grouped by depth, deepest level first: order
// (device) lists node indices, level_off (host) the start of each level in it
struct RefitPlan {
  int* order = nullptr;
  std::vector<int> level_off;
};
// rewrites the stream and shading records from new triangles (device) and, with
// refit_nodes, every child box level by level and the scene box (root_out: lo, hi)
int launch_refit(const RefitPlan& plan, const yc_triangle* tris_dev, int n_tri, float4* nodes, float4* stream,
                 int n_slots, float4* shade, bool wide, int root_link, bool refit_nodes, float4* root_out,
                 cudaStream_t s);

// widen.cu: the four-child walk index of a two-child hierarchy whose root is node 0. The
// plan finds the wide nodes (their number, and the stack entries a walk over them can need)
// in `tmp` (widen_tmp_ints ints), the write fills them in (8 float4 each), and after a refit of
// the two-child nodes widen_boxes copies their boxes over again. A small hierarchy's index is
// one launch: `wide` takes n_nodes nodes at most, ctl[0] the stack entries, ctl[1] the nodes.
bool widen_in_one_launch(int n_nodes);
cudaError_t widen_small(const float4* n2, int n_nodes, float4* wide, int* ctl, cudaStream_t s);
size_t widen_tmp_ints(int n_nodes);
cudaError_t widen_plan(const float4* n2, int n_nodes, int* tmp, int& n_wide, int& need, cudaStream_t s);
cudaError_t widen_write(const float4* n2, int n_nodes, const int* tmp, float4* wide, cudaStream_t s);
cudaError_t widen_boxes(const float4* n2, float4* wide, int n_wide, cudaStream_t s);
// bvh_build.cu: exclusive scan of n ints; tile_sum: one int per 1024
void launch_exclusive_scan(const int* in, int* out, int* tile_sum, int n, cudaStream_t s);

// launchers (udpt.cu / trace.cu)
void launch_raygen(const PassParams& pp, const PathState& ps, int* q_closest, RoundCounters* rc, DevStats* st,
                   cudaStream_t s);
// appends the next passes of the paths in pp.q_restart
void launch_raygen_next(const PassParams& pp, const PathState& ps, int* q_closest, RoundCounters* rc, DevStats* st,
                        int grid, cudaStream_t s);
// sorted/sctl: the round's shade queue (the paths of the closest-hit and the waiting queue) sorted
// by phase and material class, used when sctl->use is set (null: the queues in order)
void launch_logic(const PassParams& pp, const PathState& ps, const int* in_closest, const int* in_wait,
                  const RoundCounters* rc_in, int* out_closest, int* out_wait, int* q_any, RoundCounters* rc_out,
                  DevStats* st, int grid, cudaStream_t s, const int* sorted = nullptr,
                  const SortCtl* sctl = nullptr);
// a round's closest-hit queue alone, and its segments alone (whole stack in shared memory)
int launch_trace(const DevScene& sc, const int* queue, RoundCounters* rc, const PathState& ps, DevStats* st,
                 int grid_blocks, cudaStream_t s);
int launch_trace_segments(const DevScene& sc, const int* q_any, RoundCounters* rc, const Segments& sg, DevStats* st,
                          int grid_blocks, cudaStream_t s);
void launch_tonemap(const float4* in, float4* out, int n, cudaStream_t s);
// tail.cu: finish a pass's paths one thread each once at most `threshold` are left
int tail_capacity(const PassParams& pp, int n_smem, int* grid_out);
// n_smem, spill: as for launch_trace_mixed (grid * TAIL_TB columns)
int launch_tail(const PassParams& pp, const PathState& ps, const int* in_closest, const int* in_wait,
                RoundCounters* rc_in, int threshold, DevStats* st, int grid, cudaStream_t s, int n_smem, int* spill);
// direct query: rays as 9 floats each
// (n_smem, spill: as for launch_trace_mixed)
int launch_trace_rays(const DevScene& sc, bool any_hit, const float* rays9, int n, int* tri_out, float* t_out,
                      int* work, DevStats* st, int grid_blocks, cudaStream_t s, int n_smem, int* spill);
int trace_rays_grid_blocks(const DevScene& sc, bool any_hit, int n, int n_smem);
int trace_grid_blocks(bool any_hit, int depth, bool wide);
// one launch over both queues of a round (closest-hit entries, then any-hit); the work
// cursor is rc->work_closest. n_smem (< the stack depth, with spill): walk-stack entries in
// shared memory, the deeper ones in `spill` (grid_blocks * TRACE_TB columns of
// 2 * (depth - n_smem) ints); otherwise the whole stack is in shared memory.
int launch_trace_mixed(const DevScene& sc, const int* q_closest, const int* q_any, RoundCounters* rc,
                       const PathState& ps, const Segments& sg, DevStats* st, int grid_blocks, cudaStream_t s,
                       const int* sorted = nullptr, const RaySortCtl* rs = nullptr, int n_smem = 0,
                       int* spill = nullptr);
// raysort.cu: sorts the round's work list (closest-hit queue, then any-hit queue) into
// b.sorted when the round has at least b.threshold rays, and sets b.ctl->use
int raysort_bins(int ob, int db, int jb = 0);
int launch_raysort(const DevScene& sc, const int* q_closest, const int* q_any, const RoundCounters* rc,
                   SF<float4> ro, SF<float4> rd, const RaySortBufs& b, int grid, cudaStream_t s,
                   const Segments& sg);
int trace_mixed_grid_blocks(int depth, bool wide, int n_smem = 0);
int trace_stack_cap(int depth);   // walk-stack entries the per-pass kernels give a scene of this depth
constexpr int TRACE_TB_PASS = 128;   // block of the per-pass trace kernels (TRACE_TB of yc_trace_loop.cuh)
int l2_read_gbs(size_t bytes, int iters, cudaStream_t s, double* gbs);
// bvh_build.cu: BVH::createBVH on the device (the node array of the host builder)
// too_deep: the tree would pass 1024 levels (more than leaf_max triangles with one centroid)
cudaError_t bvh_build_device(const yc_triangle* tris_dev, int n, int bins, int leaf_max, cudaStream_t s,
                             std::vector<yc_bvh_node>& out, int& depth, bool& too_deep);

}  // namespace yc
