// A CUDA runtime without a device, for tests of the library's host code: memory is host memory, launches (fake_launch.cu) run
// nothing.  Loaded, under the runtime's soname, before libpbg_b200.so.
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

static cudaError_t last = cudaSuccess;               // kept until cudaGetLastError asks for it

extern "C" {
const char *fake_kernel_name(const void *);
cudaError_t fake_refuse(cudaError_t e) { return last = e; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int) {
  const char *name = getenv("FAKE_REFUSED");       // a kernel that the device cannot hold
  return name && strstr(fake_kernel_name(f), name) ? fake_refuse(cudaErrorInvalidValue) : cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
char __cudaInitModule(void **) { return 1; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }

static bool no_memory = false;
void fake_no_memory(int yes) { no_memory = yes != 0; }
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = nullptr;
  if (no_memory || posix_memalign(p, 256, n ? n : 1)) return fake_refuse(cudaErrorMemoryAllocation);
  memset(*p, 0xA5, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (!d || !s) return fake_refuse(cudaErrorInvalidValue);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) { static char scratch[1 << 22]; *p = scratch; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) { *n = getenv("FAKE_NO_CLUSTERS") ? 0 : 8; return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
static int fake_encode() { return 0; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **p, unsigned long long, cudaDriverEntryPointQueryResult *q) {
  *p = (void *)fake_encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}
