// A CUDA runtime without a GPU, for tests of the library's host code: loaded
// ahead of the real one (LD_PRELOAD).  Device memory is host memory, copies are
// made at once, streams, events and graphs are empty handles, and a kernel
// launch is only counted.  fake_fail_allocations(k) makes the k-th
// cudaMallocAsync from then on fail, and those after it (0: none);
// fake_launches() is the number of launches so far, fake_last_grid() the CTAs of
// the last one, fake_copies() that of cudaMemcpyAsync calls, fake_live() the
// cudaMallocAsync allocations not yet freed;
// fake_capturing(1) has streams report that they are being captured.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>

static long g_launches = 0, g_fail_at = 0, g_allocs = 0, g_grid = 0, g_live = 0, g_copies = 0;
static int g_capturing = 0;

extern "C" {

void fake_fail_allocations(long k) {
  g_fail_at = k;
  g_allocs = 0;
}
long fake_launches() { return g_launches; }
long fake_last_grid() { return g_grid; }
long fake_live() { return g_live; }
long fake_copies() { return g_copies; }
void fake_capturing(int on) { g_capturing = on; }

static cudaError_t give(void **p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
static cudaError_t launched(dim3 g) {
  ++g_launches;
  g_grid = (long)g.x * g.y * g.z;
  return cudaSuccess;
}

cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) {
  if (g_fail_at && ++g_allocs >= g_fail_at) return cudaErrorMemoryAllocation;
  ++g_live;
  return give(p, n);
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
  --g_live;
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return give(p, n); }
cudaError_t cudaFree(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return give(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return give(p, n); }
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  ++g_copies;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void *, dim3 g, dim3, void **, size_t, cudaStream_t) {
  return launched(g);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) {
  return launched(c->gridDim);
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *n, void *s) {
  *g = *b = dim3(1, 1, 1);
  *n = 0;
  *(void **)s = nullptr;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
  static void *handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *,
                            dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory" : "error";
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                   unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorInvalidSymbol; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **, unsigned long long,
                                    cudaDriverEntryPointQueryResult *) {
  return cudaErrorNotSupported;
}

static int g_handle;
cudaError_t cudaStreamCreate(cudaStream_t *s) {
  *s = (cudaStream_t)&g_handle;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return cudaStreamCreate(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
  *st = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = (cudaGraph_t)&g_handle;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long) {
  *g = (cudaGraphExec_t)&g_handle;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return launched(dim3(1, 1, 1)); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)&g_handle;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}

}  // extern "C"
