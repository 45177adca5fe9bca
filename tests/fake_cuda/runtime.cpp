// A CUDA runtime without a device, for tests of the library's host code: device memory is host
// memory up to a limit that a test sets, an allocation above it fails as cudaMalloc does when
// the device is full, copies are copies, and kernels do not run (each launch is counted). A
// render of this runtime ends at its first look at the (empty) queues.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>

namespace {
std::map<void*, size_t> g_live;
size_t g_bytes = 0, g_peak = 0, g_limit = ~(size_t)0;
long long g_launches = 0, g_mallocs = 0;
cudaError_t g_last = cudaSuccess;
int g_handle;   // what streams, events and graphs point to

cudaError_t error(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
template <class T>
cudaError_t handle(T* out) {
  *out = reinterpret_cast<T>(&g_handle);
  return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- what a test sets and reads ----
void fake_limit(unsigned long long bytes) { g_limit = bytes; }
unsigned long long fake_bytes(void) { return g_bytes; }
unsigned long long fake_peak(void) { return g_peak; }
void fake_reset_peak(void) { g_peak = g_bytes; }
long long fake_launches(void) { return g_launches; }
long long fake_mallocs(void) { return g_mallocs; }   // calls so far
int fake_allocations(void) { return (int)g_live.size(); }   // in place now

// what kernels would have left: int `at` of every allocation of exactly this many bytes
void fake_store(unsigned long long bytes, int at, int value) {
  for (const auto& a : g_live)
    if (a.second == bytes) static_cast<int*>(a.first)[at] = value;
}

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  ++g_mallocs;
  if (g_bytes + n > g_limit) return error(cudaErrorMemoryAllocation);
  *p = std::calloc(n ? n : 1, 1);
  g_live[*p] = n;
  g_bytes += n;
  if (g_bytes > g_peak) g_peak = g_bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  const auto it = g_live.find(p);
  if (it == g_live.end()) return p ? error(cudaErrorInvalidValue) : cudaSuccess;
  g_bytes -= it->second;
  g_live.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  *p = nullptr;
  return error(cudaErrorInvalidValue);
}

// ---- device, errors ----
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t smem, unsigned) {
  const size_t fit = (227 << 10) / (smem + 1024);
  *n = fit > 4 ? 4 : (int)fit;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError(void) { return g_last; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { return handle(x); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.0f, cudaSuccess; }

// ---- what the compiler's host code calls ----
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) {
  ++g_launches;
  return cudaSuccess;
}

}  // extern "C"
