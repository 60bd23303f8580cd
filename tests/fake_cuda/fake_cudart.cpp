// A CUDA runtime without a GPU, for tests of the host code's error paths: the
// library's objects are linked against it instead of the real one.
//
// Device memory is host memory filled with 0x3f bytes (doubles of 4.7e-4),
// copies and fills are done at once, kernels do nothing.  The k-th call after
// fake_arm(k) that a runtime can refuse (allocations, copies, launches, events,
// waits) returns an error.  Streams, events and waits are followed by vector
// clocks (fake_null_stream(): operations on the null stream): memory freed on a stream that is not ordered after the work of the
// others is counted in fake_violations(), and fake_in_flight() counts the
// streams whose work the host has not waited for.  fake_missed(): a copy or
// launch was refused in the call sequence before the last fake_arm and no copy
// of that size, or launch of that kernel, was made since.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

namespace {

using Clock = std::map<const void *, long long>;
void merge(Clock &a, const Clock &b) {
  for (auto &e : b) a[e.first] = std::max(a[e.first], e.second);
}

std::map<const void *, Clock> g_after;  // per stream: what its next work is ordered after, its own included
Clock g_host;                           // what the host has waited for
std::map<const void *, Clock> g_event;
long long g_calls, g_fail_at, g_launches, g_next = 1;
long long g_violations;
cudaError_t g_last = cudaSuccess;

size_t g_refused, g_missing;  // a kernel's address or a copy's size
std::set<size_t> g_done;

cudaError_t refuse(size_t what = 0) {
  if (++g_calls != g_fail_at) return cudaSuccess;
  g_refused = what;
  return g_last = cudaErrorUnknown;
}
cudaError_t work(const void *st, size_t what = 0) {
  cudaError_t e = refuse(what);
  if (e != cudaSuccess) return e;
  g_after[st][st]++;
  g_done.insert(what);
  return e;
}
void *fresh() { return reinterpret_cast<void *>(0x1000 + 16 * g_next++); }
struct Config {
  dim3 grid, block;
  size_t smem;
  void *stream;
} g_config;

}  // namespace

extern "C" {

void fake_arm(long long k) {
  g_calls = 0, g_fail_at = k, g_launches = 0, g_last = cudaSuccess;
  g_missing = g_refused, g_refused = 0;
  g_done.clear();
}
int fake_missed() { return g_missing && !g_done.count(g_missing); }
long long fake_calls() { return g_calls; }
long long fake_launches() { return g_launches; }
long long fake_violations() { return g_violations; }
long long fake_null_stream() { return g_after[nullptr][nullptr]; }
long long fake_in_flight() {
  long long n = 0;
  for (auto &s : g_after)
    for (auto &e : s.second) n += e.second > g_host[e.first];
  return n;
}

cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) { return *p = (cudaMemPool_t)fresh(), cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void *) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

cudaError_t cudaMalloc(void **p, size_t n) {
  const cudaError_t e = refuse();
  if (e != cudaSuccess) return e;
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  std::memset(*p, 0x3f, n);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *) { return cudaSuccess; }  // (kept: a late reader is counted, not crashed)
cudaError_t cudaFreeAsync(void *, cudaStream_t st) {
  for (auto &s : g_after)
    for (auto &e : s.second)
      if (e.second > g_host[e.first] && e.second > g_after[st][e.first]) {
        g_violations++;
        return cudaSuccess;
      }
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind, cudaStream_t st) {
  const cudaError_t e = work(st, n);
  if (e == cudaSuccess) std::memcpy(d, s, n);
  return e;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  const cudaError_t e = work(st);
  if (e == cudaSuccess) std::memset(d, v, n);
  return e;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return *p = fresh(), cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *st, unsigned) {
  const cudaError_t e = refuse();
  if (e == cudaSuccess) *st = (cudaStream_t)fresh();
  return e;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) { return merge(g_host, g_after[st]), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t ev, unsigned) {
  const cudaError_t e = refuse();
  if (e == cudaSuccess) merge(g_after[st], g_event[ev]);
  return e;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *ev, unsigned) {
  const cudaError_t e = refuse();
  if (e == cudaSuccess) *ev = (cudaEvent_t)fresh();
  return e;
}
cudaError_t cudaEventCreate(cudaEvent_t *ev) { return cudaEventCreateWithFlags(ev, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t st) {
  const cudaError_t e = refuse();
  if (e == cudaSuccess) g_event[ev] = g_after[st];
  return e;
}
cudaError_t cudaEventSynchronize(cudaEvent_t ev) { return merge(g_host, g_event[ev]), cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void *, enum cudaFuncAttribute, int) { return refuse(); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  return *n = 2, cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  g_launches++;
  return work(c->stream, (size_t)f);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *st) {
  g_config = {grid, block, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
  *grid = g_config.grid, *block = g_config.block, *smem = g_config.smem, *(void **)st = g_config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { return *k = (cudaKernel_t)f, cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t f, dim3, dim3, void **, size_t, cudaStream_t st) {
  g_launches++;
  return work(st, (size_t)f);
}
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

// (graphs: the host-buffer pipeline, which these tests do not take)
cudaError_t cudaGraphCreate(cudaGraph_t *, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphAddEmptyNode(cudaGraphNode_t *, cudaGraph_t, const cudaGraphNode_t *, size_t) {
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t *, cudaGraph_t, const cudaGraphNode_t *, size_t,
                                   const struct cudaKernelNodeParams *) {
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphAddMemcpyNode1D(cudaGraphNode_t *, cudaGraph_t, const cudaGraphNode_t *, size_t, void *,
                                     const void *, size_t, enum cudaMemcpyKind) {
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
}
