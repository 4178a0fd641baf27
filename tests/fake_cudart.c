/* A CUDA runtime in host memory for tests without a GPU: preloaded before
 * libcudart, it replaces the calls that a context's creation and its reads of
 * values make.  Kernels do not run.  It counts the bytes copied to the host
 * and can refuse those copies or the synchronisation after them. */
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

#define API __attribute__((visibility("default")))
enum { kOk = 0, kInvalidValue = 1, kUnknown = 999, kDeviceToHost = 2 };

static size_t d2h_bytes, d2h_copies;
static int fail_copy, fail_sync;

API size_t fake_d2h_bytes(void) { return d2h_bytes; }
API size_t fake_d2h_copies(void) { return d2h_copies; }
API void fake_reset(int copy, int sync) {
  d2h_bytes = d2h_copies = 0;
  fail_copy = copy;
  fail_sync = sync;
}

API int cudaSetDevice(int d) { return d == 0 ? kOk : kInvalidValue; }
API int cudaGetDevice(int* d) { return *d = 0, kOk; }
API int cudaGetLastError(void) { return kOk; }
API int cudaDeviceGetAttribute(int* v, int a, int d) { return (void)a, (void)d, *v = 1, kOk; }
API int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned fl) {
  return (void)f, (void)b, (void)s, (void)fl, *n = 0, kOk;
}
API int cudaStreamCreateWithFlags(void** s, unsigned f) { return (void)f, *s = malloc(1), kOk; }
API int cudaStreamDestroy(void* s) { return free(s), kOk; }
API int cudaStreamSynchronize(void* s) { return (void)s, fail_sync ? kUnknown : kOk; }
API int cudaEventCreate(void** e) { return *e = malloc(1), kOk; }
API int cudaEventCreateWithFlags(void** e, unsigned f) { return (void)f, *e = malloc(1), kOk; }
API int cudaEventDestroy(void* e) { return free(e), kOk; }
API int cudaMalloc(void** p, size_t n) { return *p = calloc(n ? n : 1, 1), *p ? kOk : 2; }
API int cudaFree(void* p) { return free(p), kOk; }
API int cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), kOk; }
API int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) {
  (void)st;
  if (kind == kDeviceToHost) {
    if (fail_copy) return kUnknown;
    d2h_bytes += n;
    ++d2h_copies;
  }
  memcpy(d, s, n);
  return kOk;
}
API int cudaMemcpy(void* d, const void* s, size_t n, int kind) { return cudaMemcpyAsync(d, s, n, kind, NULL); }
API int cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, int kind, void* st) {
  int rc = kOk;
  for (size_t i = 0; i < h && rc == kOk; ++i)
    rc = cudaMemcpyAsync((char*)d + i * dp, (const char*)s + i * sp, w, kind, st);
  return rc;
}
API int cudaLaunchKernel(const void* f, ...) { return (void)f, kOk; }
API int cudaLaunchKernelExC(const void* c, const void* f, void** a) { return (void)c, (void)f, (void)a, kOk; }
