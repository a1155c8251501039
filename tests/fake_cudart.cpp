// A CUDA runtime without a GPU for tests of the library's host code: device memory is
// host memory, kernels do nothing, and every stream keeps a clock of the work that
// precedes its tail, so that a test can ask which work nobody has waited for.  The
// n-th call that may fail can be made to (fake_fail_at).
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>

namespace {
using Clock = std::map<void *, long long>;
std::map<void *, Clock> streams;  // of the work before each stream's tail; null: the default
std::map<void *, Clock> events;
Clock issued, done;
std::set<void *> live_streams, live_events, live_mem;
long long calls = 0, fail_at = 0;
cudaError_t last = cudaSuccess;

cudaError_t step() {
  if (fail_at > 0 && ++calls == fail_at) return last = cudaErrorUnknown;
  return cudaSuccess;
}
void join(Clock &a, const Clock &b) {
  for (auto &p : b)
    if (p.second > a[p.first]) a[p.first] = p.second;
}
cudaError_t work(void *s) {
  const cudaError_t e = step();
  if (!e) streams[s][s] = ++issued[s];
  return e;
}
cudaError_t mem(void **p, size_t n) {
  const cudaError_t e = step();
  if (e) return last = cudaErrorMemoryAllocation;
  *p = std::calloc(n ? n : 1, 1);
  live_mem.insert(*p);
  return cudaSuccess;
}
cudaError_t gone(void *p) {
  if (p && live_mem.erase(p)) std::free(p);
  return cudaSuccess;
}
cudaError_t new_stream(cudaStream_t *s) {
  const cudaError_t e = step();
  if (!e) live_streams.insert(*s = (cudaStream_t)std::malloc(1));
  return e;
}
cudaError_t new_event(cudaEvent_t *v) {
  const cudaError_t e = step();
  if (!e) live_events.insert(*v = (cudaEvent_t)std::malloc(1));
  return e;
}
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
cudaStream_t cfg_stream;
}  // namespace

extern "C" {
void fake_fail_at(long long n) {
  fail_at = n;
  calls = 0;
  last = cudaSuccess;
}
int fake_pending() {  // streams with work that nobody has waited for
  int n = 0;
  for (auto &p : issued) n += p.second > done[p.first];
  return n;
}
int fake_live(int what) {
  return (int)(what == 0 ? live_streams : what == 1 ? live_events : live_mem).size();
}

unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void *s) {
  cfg_grid = g;
  cfg_block = b;
  cfg_smem = m;
  cfg_stream = (cudaStream_t)s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
  *g = cfg_grid;
  *b = cfg_block;
  *m = cfg_smem;
  *(cudaStream_t *)s = cfg_stream;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { return (void **)&calls; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t s) {
  return work(s);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { return *a = 0, *b = -5, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
  done = issued;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
  std::memset(a, 0, sizeof *a);
  a->ptxVersion = a->binaryVersion = 100;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return step(); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                   unsigned) {
  return *n = 1, cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *, void **, unsigned long long,
                                    cudaDriverEntryPointQueryResult *) {
  return cudaErrorUnknown;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorUnknown; }

cudaError_t cudaMalloc(void **p, size_t n) { return mem(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return mem(p, n); }
cudaError_t cudaFree(void *p) { return gone(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return gone(p); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  const cudaError_t e = step();
  if (!e) std::memcpy(d, s, n);
  return e;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  const cudaError_t e = work(st);
  if (!e) std::memcpy(d, s, n);
  return e;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  const cudaError_t e = step();
  if (!e) std::memset(p, v, n);
  return e;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
  const cudaError_t e = work(s);
  if (!e) std::memset(p, v, n);
  return e;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return new_stream(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return new_stream(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  live_streams.erase(s);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) {
  return *c = cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  join(done, streams[s]);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t v, unsigned) {
  const cudaError_t e = step();
  if (!e) join(streams[s], events[v]);
  return e;
}
cudaError_t cudaEventCreate(cudaEvent_t *v) { return new_event(v); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *v, unsigned) { return new_event(v); }
cudaError_t cudaEventDestroy(cudaEvent_t v) {
  live_events.erase(v);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t v, cudaStream_t s) {
  const cudaError_t e = step();
  if (!e) events[v] = streams[s];
  return e;
}
cudaError_t cudaEventSynchronize(cudaEvent_t v) {
  join(done, events[v]);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { return *t = 0.f, cudaSuccess; }

// the dense solver's library, not used here
int cusolverDnCreate() { return 1; }
int cusolverDnCreateParams() { return 1; }
int cusolverDnDestroy() { return 1; }
int cusolverDnDestroyParams() { return 1; }
int cusolverDnSetStream() { return 1; }
int cusolverDnXgetrf() { return 1; }
int cusolverDnXgetrf_bufferSize() { return 1; }
int cusolverDnXgetrs() { return 1; }
}
