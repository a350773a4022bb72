// A CUDA runtime without a GPU, preloaded by tests/test_failed_loading.py: device
// memory is zeroed host memory, copies happen at once, kernels are counted and
// not run.  The n-th allocation from now on, or all from then on, can be made to fail.
#include <stdlib.h>
#include <string.h>

#define CUDA_OK 0
#define CUDA_NO_MEMORY 2
static long fail_in = -1, fail_all = 0, launches = 0, live = 0;

// Lets n allocations pass and fails the next one (n < 0: none).
void fake_fail_after(long n) { fail_in = n, fail_all = 0; }
// The same, and fails every later one too.
void fake_fail_from(long n) { fail_in = n, fail_all = 1; }
long fake_launches(void) { return launches; }
long fake_live(void) { return live; }

static int take(void **p, size_t n) {
  *p = 0;
  if (fail_in == 0) {
    if (!fail_all) fail_in = -1;
    return CUDA_NO_MEMORY;
  }
  if (fail_in > 0) --fail_in;
  *p = calloc(1, n ? n : 1);
  ++live;
  return CUDA_OK;
}
static int give(void *p) {
  if (p) --live;
  free(p);
  return CUDA_OK;
}
static int handle(void **p) {
  *p = malloc(1);
  return CUDA_OK;
}

int cudaMalloc(void **p, size_t n) { return take(p, n); }
int cudaHostAlloc(void **p, size_t n, unsigned flags) { return (void)flags, take(p, n); }
int cudaFree(void *p) { return give(p); }
int cudaFreeHost(void *p) { return give(p); }
int cudaMemcpyAsync(void *dst, const void *src, size_t n, int kind, void *st) {
  (void)kind, (void)st;
  memcpy(dst, src, n);
  return CUDA_OK;
}
int cudaMemsetAsync(void *p, int v, size_t n, void *st) {
  (void)st;
  memset(p, v, n);
  return CUDA_OK;
}
int cudaLaunchKernelExC(const void *cfg, const void *f, void **args) {
  (void)cfg, (void)f, (void)args;
  ++launches;
  return CUDA_OK;
}
struct dim3_ { unsigned x, y, z; };
int cudaLaunchKernel(const void *f, struct dim3_ g, struct dim3_ b, void **args, size_t s,
                     void *st) {
  (void)f, (void)g, (void)b, (void)args, (void)s, (void)st;
  ++launches;
  return CUDA_OK;
}
int cudaFuncSetAttribute(const void *f, int a, int v) { return (void)f, (void)a, (void)v, CUDA_OK; }
int cudaGetDeviceCount(int *n) { return *n = 1, CUDA_OK; }
int cudaSetDevice(int d) { return (void)d, CUDA_OK; }
int cudaGetDevice(int *d) { return *d = 0, CUDA_OK; }
int cudaDeviceGetAttribute(int *v, int a, int d) { return (void)a, (void)d, *v = 148, CUDA_OK; }
int cudaStreamCreateWithFlags(void **s, unsigned f) { return (void)f, handle(s); }
int cudaStreamDestroy(void *s) { return free(s), CUDA_OK; }
int cudaStreamSynchronize(void *s) { return (void)s, CUDA_OK; }
int cudaGetLastError(void) { return CUDA_OK; }
