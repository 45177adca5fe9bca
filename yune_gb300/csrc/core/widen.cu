// widen.cu -- the four-child walk index of an uploaded two-child hierarchy.
//
// The two-child nodes over the reference's leaves (tree mode 1, yc_scene.h) stay the
// scene's layout: they are what the upload writes, what the digest covers and what a refit
// recomputes. The traversal kernels walk this index instead, the same hierarchy with up to
// four children per node, made here on the device after the upload. A walk's time follows
// the number of nodes it opens one after another (each a dependent fetch and a step that
// the warp's lanes take in turn) more than the number of boxes it tests: four-child nodes
// take 12 visits where two-child nodes take 27 (glass sphere, closest-hit rays) for 12% fewer
// boxes. Traversal of one 1920x1080 pass of a 260K-triangle scene: 4.10 ms over the
// two-child nodes, 3.26 ms over the index; glass sphere 1024x1024 3.36 -> 2.90 ms;
// 758K-triangle field 9.9 -> 8.5 ms.
//
// A wide node replaces a two-child node and the descendants opened into it: its two children
// first, then, while there is room, the largest interior child by surface area is replaced
// by its own two. The set of two-child nodes that become wide nodes is found level by level
// from the root (k_widen_level marks them), an exclusive scan of the marks numbers the wide
// nodes in the order of the two-child array (pre-order, so a subtree stays together), and one
// launch writes them. Every child box is a copy of the two-child node's, so the boxes
// a ray has to pass on its way to a leaf are a subset of those of the two-child walk, ending
// with the leaf's own.
#include <cuda_runtime.h>

#include <algorithm>

#include "yc_internal.h"

namespace yc {

namespace {

constexpr int WIDEN_TB = 256;
constexpr int WIDEN_LEVELS = 16;   // levels launched between two looks at the frontier

// one child of a wide node: the two-child node that holds its box and which of the two
struct Kid {
  int src;      // 2 * node + side
  int link;
  float area;   // of an interior child; -1 for a leaf (never opened)
};

__device__ __forceinline__ Kid kid_of(const float4* __restrict__ n2, int node, int side) {
  const float4* nd = n2 + 4 * (size_t)node;
  const int2 l = __ldg(reinterpret_cast<const int2*>(nd + 3));
  Kid k{2 * node + side, side ? l.y : l.x, -1.0f};
  if (k.link >= 0) {
    const float4 x = __ldg(nd), y = __ldg(nd + 1), z = __ldg(nd + 2);
    const float dx = side ? x.w - x.y : x.z - x.x, dy = side ? y.w - y.y : y.z - y.x, dz = side ? z.w - z.y : z.z - z.x;
    k.area = dx * dy + dy * dz + dz * dx;
  }
  return k;
}

// the children of the wide node in place of two-child node `node`; returns how many
__device__ __forceinline__ int pick_kids(const float4* __restrict__ n2, int node, Kid (&kid)[4]) {
  kid[0] = kid_of(n2, node, 0);
  kid[1] = kid_of(n2, node, 1);
  kid[2] = kid[3] = Kid{-1, LINK_NONE, -1.0f};
  int n = 2;
#pragma unroll
  for (int round = 0; round < 2; ++round) {
    int at = -1;
    float best = -1.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c < n && kid[c].link >= 0 && (at < 0 || kid[c].area > best)) { best = kid[c].area; at = c; }
    if (at < 0) break;
    int open = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c == at) open = kid[c].link;
    const Kid a = kid_of(n2, open, 0), b = kid_of(n2, open, 1);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c == at) kid[c] = a;
      if (c == n) kid[c] = b;
    }
    ++n;
  }
  return n;
}

// One level: every two-child node of the frontier becomes a wide node, its interior
// children the next frontier. A frontier entry carries the stack entries a walk can hold when it
// arrives there; *need receives the most a walk can hold anywhere.
__global__ void __launch_bounds__(WIDEN_TB) k_widen_level(const float4* __restrict__ n2, int n_nodes,
                                                          const int2* __restrict__ in, const int* n_in, int2* out,
                                                          int* n_out, int* mark, int* need) {
  const int n = *n_in;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int2 f = in[i];
    mark[f.x] = 1;
    Kid kid[4];
    const int held = f.y + pick_kids(n2, f.x, kid) - 1;
    atomicMax(need, held);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (kid[c].link >= 0 && kid[c].link < n_nodes) out[atomicAdd(n_out, 1)] = make_int2(kid[c].link, held);
  }
}

__global__ void k_widen_root(int2* frontier) { *frontier = make_int2(0, 0); }

// the box of child c from the two-child node that holds it; an empty slot (src < 0, a link of
// LINK_NONE) gets an inverted one
__device__ __forceinline__ void put_box(float (&v)[6][4], int c, const float4* __restrict__ n2, int src) {
  const float INF = __int_as_float(0x7f800000);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float lo = INF, hi = -INF;
    if (src >= 0) {
      const float4 q = __ldg(n2 + 4 * (size_t)(src >> 1) + k);
      lo = (src & 1) ? q.y : q.x;
      hi = (src & 1) ? q.w : q.z;
    }
    v[2 * k][c] = lo;
    v[2 * k + 1][c] = hi;
  }
}

__device__ __forceinline__ void store_boxes(float4* o, const float (&v)[6][4]) {
#pragma unroll
  for (int f = 0; f < 6; ++f) o[f] = make_float4(v[f][0], v[f][1], v[f][2], v[f][3]);
}

// the wide node of two-child node i (yc_scene.h); its last 16 bytes hold its children's src,
// for refits
__device__ __forceinline__ void write_wide(const float4* __restrict__ n2, int i, const int* slot, float4* wide) {
  Kid kid[4];
  pick_kids(n2, i, kid);
  float v[6][4];
  int link[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    put_box(v, c, n2, kid[c].src);
    link[c] = kid[c].link >= 0 && kid[c].link != LINK_NONE ? slot[kid[c].link] : kid[c].link;
  }
  float4* o = wide + 8 * (size_t)slot[i];
  store_boxes(o, v);
  reinterpret_cast<int4*>(o)[6] = make_int4(link[0], link[1], link[2], link[3]);
  reinterpret_cast<int4*>(o)[7] = make_int4(kid[0].src, kid[1].src, kid[2].src, kid[3].src);
}

__global__ void __launch_bounds__(WIDEN_TB) k_widen_write(const float4* __restrict__ n2, int n_nodes,
                                                          const int* __restrict__ mark, const int* __restrict__ slot,
                                                          float4* wide) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_nodes && mark[i]) write_wide(n2, i, slot, wide);
}

// The whole index of a hierarchy of at most WIDEN_SMALL nodes in one block: the levels, the
// numbering and the nodes (the launches and copies of the general path cost 0.15 ms, a tenth of
// a small scene's upload). ctl: the stack entries a walk can need, the number of wide nodes.
constexpr int WIDEN_SMALL = 2048;
constexpr int SMALL_TB = 1024;
static_assert(WIDEN_SMALL == 2 * SMALL_TB, "a thread numbers two nodes");

__global__ void __launch_bounds__(SMALL_TB) k_widen_small(const float4* __restrict__ n2, int n_nodes, float4* wide,
                                                          int* ctl) {
  __shared__ int s_slot[WIDEN_SMALL];              // marks, then slots
  __shared__ int2 s_front[2][WIDEN_SMALL / 2 + 1]; // (the nodes of a level are disjoint subtrees' roots)
  __shared__ int s_n[2], s_need, s_warp[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < WIDEN_SMALL; i += SMALL_TB) s_slot[i] = 0;
  if (tid == 0) {
    s_front[0][0] = make_int2(0, 0);
    s_n[0] = 1;
    s_need = 0;
  }
  __syncthreads();
  for (int cur = 0;; cur ^= 1) {
    const int n = s_n[cur];
    __syncthreads();
    if (n == 0) break;
    if (tid == 0) s_n[cur ^ 1] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += SMALL_TB) {
      const int2 f = s_front[cur][i];
      s_slot[f.x] = 1;
      Kid kid[4];
      const int held = f.y + pick_kids(n2, f.x, kid) - 1;
      atomicMax(&s_need, held);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (kid[c].link >= 0 && kid[c].link < n_nodes) {
          const int at = atomicAdd(&s_n[cur ^ 1], 1);
          if (at <= WIDEN_SMALL / 2) s_front[cur ^ 1][at] = make_int2(kid[c].link, held);
        }
    }
    __syncthreads();
  }
  // the slots: an exclusive scan of the marks, two per thread
  const int m0 = s_slot[2 * tid], m1 = s_slot[2 * tid + 1];
  int incl = m0 + m1;
  for (int off = 1; off < 32; off <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += u;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int v = s_warp[lane];
    for (int off = 1; off < 32; off <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, off);
      if (lane >= off) v += u;
    }
    s_warp[lane] = v;
  }
  __syncthreads();
  const int before = incl - m0 - m1 + (warp > 0 ? s_warp[warp - 1] : 0);
  s_slot[2 * tid] = before;
  s_slot[2 * tid + 1] = before + m0;
  __syncthreads();
  if (m0) write_wide(n2, 2 * tid, s_slot, wide);
  if (m1) write_wide(n2, 2 * tid + 1, s_slot, wide);
  if (tid == 0) {
    ctl[0] = s_need;
    ctl[1] = s_warp[31];
  }
}

// the child boxes of every wide node, again from the (refitted) two-child nodes
__global__ void __launch_bounds__(WIDEN_TB) k_widen_boxes(const float4* __restrict__ n2, float4* wide, int n_wide) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_wide) return;
  float4* o = wide + 8 * (size_t)i;
  const int4 src = reinterpret_cast<const int4*>(o)[7];
  float v[6][4];
  put_box(v, 0, n2, src.x);
  put_box(v, 1, n2, src.y);
  put_box(v, 2, n2, src.z);
  put_box(v, 3, n2, src.w);
  store_boxes(o, v);
}

int tiles_of(int n) { return (n + 1023) / 1024; }
int blocks_of(int n) { return (n + WIDEN_TB - 1) / WIDEN_TB; }

}  // namespace

bool widen_in_one_launch(int n_nodes) { return n_nodes <= WIDEN_SMALL; }

cudaError_t widen_small(const float4* n2, int n_nodes, float4* wide, int* ctl, cudaStream_t s) {
  k_widen_small<<<1, SMALL_TB, 0, s>>>(n2, n_nodes, wide, ctl);
  return cudaPeekAtLastError();
}

// the ints of `tmp`: marks, slots, scan tiles, two frontiers, the control words
size_t widen_tmp_ints(int n_nodes) {
  return (size_t)2 * n_nodes + tiles_of(n_nodes) + 1 + (size_t)4 * (n_nodes + 1) + WIDEN_LEVELS + 2;
}

cudaError_t widen_plan(const float4* n2, int n_nodes, int* tmp, int& n_wide, int& need, cudaStream_t s) {
  int2* fa = reinterpret_cast<int2*>(tmp);
  int2* fb = fa + n_nodes + 1;
  int* mark = reinterpret_cast<int*>(fb + n_nodes + 1);
  int* slot = mark + n_nodes;
  int* tiles = slot + n_nodes;
  int* ctl = tiles + tiles_of(n_nodes) + 1;   // need, then the frontier sizes of a run of levels
  int host[WIDEN_LEVELS + 2] = {0, 1};
  cudaError_t e = cudaMemsetAsync(mark, 0, (size_t)n_nodes * sizeof(int), s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(ctl, host, sizeof(host), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return e;
  k_widen_root<<<1, 1, 0, s>>>(fa);
  const int grid = std::min(blocks_of(n_nodes), 1216);
  for (;;) {
    for (int l = 0; l < WIDEN_LEVELS; ++l) {
      k_widen_level<<<grid, WIDEN_TB, 0, s>>>(n2, n_nodes, fa, ctl + 1 + l, fb, ctl + 2 + l, mark, ctl);
      std::swap(fa, fb);
    }
    e = cudaMemcpyAsync(host, ctl, sizeof(host), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    if (host[WIDEN_LEVELS + 1] == 0) break;
    host[1] = host[WIDEN_LEVELS + 1];
    for (int l = 2; l < WIDEN_LEVELS + 2; ++l) host[l] = 0;
    e = cudaMemcpyAsync(ctl, host, sizeof(host), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
  }
  need = host[0];
  launch_exclusive_scan(mark, slot, tiles, n_nodes, s);
  int last[2];
  e = cudaMemcpyAsync(&last[0], slot + n_nodes - 1, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&last[1], mark + n_nodes - 1, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  n_wide = last[0] + last[1];
  return e;
}

cudaError_t widen_write(const float4* n2, int n_nodes, const int* tmp, float4* wide, cudaStream_t s) {
  const int* mark = tmp + (size_t)4 * (n_nodes + 1);
  k_widen_write<<<blocks_of(n_nodes), WIDEN_TB, 0, s>>>(n2, n_nodes, mark, mark + n_nodes, wide);
  return cudaPeekAtLastError();
}

cudaError_t widen_boxes(const float4* n2, float4* wide, int n_wide, cudaStream_t s) {
  k_widen_boxes<<<blocks_of(n_wide), WIDEN_TB, 0, s>>>(n2, wide, n_wide);
  return cudaPeekAtLastError();
}

}  // namespace yc
