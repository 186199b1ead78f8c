/* A stand-in for the CUDA runtime calls that the library's host code makes, to be
 * preloaded on a machine without a GPU: device memory is host memory, launches do
 * nothing.  FAKE_FAIL names the calls that fail ("hostalloc", "hostmap"); with
 * FAKE_LOCKED set, callers' arrays count as page-locked.  The 7th
 * argument of a chained launch (y of the sliced kernel, the only one that the tests make) is
 * printed by its kind: "null", "mapped" (from cudaHostAlloc) or "device". */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static char *mapped_lo, *mapped_hi;
static int live_host_allocs;

static int fails(const char* what) {
  const char* f = getenv("FAKE_FAIL");
  return f && strstr(f, what) != NULL;
}

cudaError_t cudaMalloc(void** p, size_t n) { *p = calloc(1, n ? n : 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned flags) {
  (void)flags;
  if (fails("hostalloc")) return cudaErrorMemoryAllocation;
  *p = calloc(1, n);
  mapped_lo = *p;
  mapped_hi = mapped_lo + n;
  ++live_host_allocs;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); --live_host_allocs; printf("live %d\n", live_host_allocs); fflush(stdout); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned flags) {
  (void)flags;
  if (fails("hostmap")) return cudaErrorNotSupported;
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { (void)k; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)st;
  if (k == cudaMemcpyDeviceToHost) printf("copy out %zu\n", n), fflush(stdout);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { (void)s; memset(p, v, n); return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 152; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
  (void)p;
  memset(a, 0, sizeof(*a));
  a->type = getenv("FAKE_LOCKED") ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { (void)e; return "fake error"; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { (void)f; *s = (cudaStream_t)16; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int p) { (void)f; (void)p; *s = (cudaStream_t)16; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = 0; *hi = -5; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { (void)f; *e = (cudaEvent_t)16; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned fl) {
  (void)f; (void)b; (void)s; (void)fl;
  *n = 4;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* f, void** args) {
  (void)cfg;
  (void)f;
  char* y = *(char**)args[6];
  puts(!y ? "y null" : y >= mapped_lo && y < mapped_hi ? "y mapped" : "y device");
  fflush(stdout);
  return cudaSuccess;
}
