/* A CUDA runtime in host memory for tests without a GPU: preloaded before
 * libcudart, it replaces the calls that a context's creation, its sweeps and
 * its reads of values make.  Kernels do not run.  It counts the bytes copied to
 * the host and can refuse those copies or the synchronisation after them.  Time
 * is a model: a host clock that calls advance, a device clock that kernels
 * advance by a cost set per grid size, and a device that starts a launch when
 * it is through with the one before and the host has made it. */
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
/* the clocks, in us; a graph is the sum of its kernels' costs */
static double host_us, device_us, capture_us = -1;
static double cost_us[1 << 16]; /* by grid size */
static unsigned lcg;
static double noise(void) { return lcg = lcg * 1664525u + 1013904223u, (lcg >> 8) / 16777216.0; }
static double slowing, busy_us; /* the device slows by this share per us of work it has done */
static void run(double us) {
  if (capture_us >= 0) {
    capture_us += us;
    return;
  }
  device_us = (device_us > host_us ? device_us : host_us) + us * (1 + slowing * busy_us);
  busy_us += us;
}
static void* boxed(double v) { return memcpy(malloc(sizeof v), &v, sizeof v); }

API void fake_cost(int grid, double us) { cost_us[grid] = us; }
API void fake_seed(unsigned s) { lcg = s; }
API void fake_slowing(double per_us) { slowing = per_us, busy_us = 0; }

API int cudaStreamSynchronize(void* s) {
  (void)s;
  if (device_us > host_us) host_us = device_us;
  return fail_sync ? kUnknown : kOk;
}
API int cudaStreamBeginCapture(void* s, int mode) { return (void)s, (void)mode, capture_us = 0, kOk; }
API int cudaStreamEndCapture(void* s, void** g) { return (void)s, *g = boxed(capture_us), capture_us = -1, kOk; }
API int cudaGraphInstantiate(void** e, void* g, unsigned long long f) {
  return (void)f, host_us += 1000, *e = boxed(*(double*)g), kOk;
}
API int cudaGraphDestroy(void* g) { return free(g), kOk; }
API int cudaGraphExecDestroy(void* e) { return free(e), kOk; }
/* a launch takes the host 4 to 12 us */
API int cudaGraphLaunch(void* e, void* s) { return (void)s, host_us += 4 + 8 * noise(), run(*(double*)e), kOk; }
API int cudaEventCreate(void** e) { return *e = boxed(0), kOk; }
API int cudaEventCreateWithFlags(void** e, unsigned f) { return (void)f, *e = boxed(0), kOk; }
API int cudaEventDestroy(void* e) { return free(e), kOk; }
API int cudaEventRecord(void* e, void* s) {
  return (void)s, host_us += 1, *(double*)e = device_us > host_us ? device_us : host_us, kOk;
}
API int cudaEventSynchronize(void* e) { return host_us = host_us > *(double*)e ? host_us : *(double*)e, kOk; }
API int cudaEventElapsedTime(float* ms, void* a, void* b) {
  return *ms = (float)((*(double*)b - *(double*)a) * 1e-3), kOk;
}
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
API int cudaLaunchKernelExC(const void* c, const void* f, void** a) {
  const unsigned grid = *(const unsigned*)c; /* the configuration begins with gridDim.x */
  return (void)f, (void)a, run(grid < 1 << 16 ? cost_us[grid] : 0), kOk;
}
