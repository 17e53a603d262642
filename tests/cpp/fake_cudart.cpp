// fake_cudart.cpp -- a stand-in for the CUDA runtime, for tests of the library's host side
// on the CPU: device memory is host memory with a limit, kernels do not run (a hook sees
// their names and arguments instead), streams and events have nothing to wait for.
#include "fake_cudart.h"

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

namespace fake {
size_t limit = (size_t)-1, used = 0, largest = 0;
std::function<void(const std::string &, void **)> on_launch;
std::map<std::string, int> launches;
thread_local unsigned grid = 0;
int pinned = 0;
int device = 0, sms[2] = {152, 152};
static std::map<const void *, std::string> names;
static std::map<void *, size_t> blocks;
static std::recursive_mutex mu;

static cudaError_t launch(const void *func, void **args, dim3 g = dim3(0)) {
  grid = g.x;
  std::string name = "?";
  {
    std::lock_guard<std::recursive_mutex> g(mu);
    if (names.count(func)) name = names[func];
    ++launches[name];
  }
  if (on_launch && name != "?") on_launch(name, args);
  return cudaSuccess;
}
}  // namespace fake

using namespace fake;
static thread_local int capturing = 0;

extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
  names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
static thread_local struct { dim3 g, b; size_t m; void *s; } call;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void *s) { call = {g, b, m, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
  *g = call.g; *b = call.b; *m = call.m; *(void **)s = call.s;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void **args, size_t, cudaStream_t) { return launch(k, args, g); }
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3, void **args, size_t, cudaStream_t) { return launch(f, args, g); }

cudaError_t cudaMalloc(void **p, size_t n) {
  std::lock_guard<std::recursive_mutex> g(mu);
  if (used + n > limit) return cudaErrorMemoryAllocation;
  *p = calloc(1, n);
  blocks[*p] = n;
  used += n;
  largest = n > largest ? n : largest;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::recursive_mutex> g(mu);
  if (!p) return cudaSuccess;
  if (!blocks.count(p)) abort();  // freed twice, or never allocated
  used -= blocks[p];
  blocks.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { ++pinned; *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *t = (size_t)284 << 30; *f = limit - used; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int d) { *v = sms[d]; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { *p = const_cast<void *>(s); return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { ++capturing; return cudaSuccess; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                                          cudaStreamCaptureMode) { ++capturing; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { --capturing; *g = (cudaGraph_t)1; return cudaSuccess; }
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus *s, unsigned long long *, cudaGraph_t *g,
                                     const cudaGraphNode_t **deps, const cudaGraphEdgeData **, size_t *n) {
  *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  if (g) *g = (cudaGraph_t)1;
  if (deps) *deps = nullptr;
  if (n) *n = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t *, const cudaGraphEdgeData *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) { *h = 1; return cudaSuccess; }
cudaError_t cudaGraphAddNode(cudaGraphNode_t *n, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                             cudaGraphNodeParams *p) {
  static cudaGraph_t body = (cudaGraph_t)2;
  *n = (cudaGraphNode_t)1;
  p->conditional.phGraph_out = &body;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { free(e); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return launch("graph", nullptr); }
}
