/* A stand-in for the CUDA runtime calls that a linear system makes, preloaded
   by tests/test_fake_device.py: device memory is host memory, nothing is run.
   A cooperative launch is refused as a device refuses it: more blocks than fit
   (one a SM of more than half its shared memory, else four), more shared memory
   than was asked for on the device at hand, or the FAKE_REFUSE'th one (0: none)
   whatever it is. */
#include <stdlib.h>
#include <string.h>

typedef struct { unsigned x, y, z; } dim3;
static int device, launches;
static struct { const void *f; int dev, bytes; } attr[256];
static int nattr;

static int env(const char *name, int dflt) {
  const char *v = getenv(name);
  return v ? atoi(v) : dflt;
}
int cudaSetDevice(int d) { device = d; return 0; }
int cudaGetDevice(int *d) { *d = device; return 0; }
int cudaGetLastError(void) { return 0; }
int cudaDeviceGetAttribute(int *v, int a, int d) { *v = a == 16 ? env("FAKE_SMS", 152) : 0; return 0; }
int cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)1 << 34; return 0; }
int cudaMalloc(void **p, size_t n) { *p = calloc(n + 256, 1); return *p ? 0 : 2; }
int cudaFree(void *p) { free(p); return 0; }
int cudaStreamCreateWithFlags(void **s, unsigned f) { *s = malloc(1); return 0; }
int cudaStreamDestroy(void *s) { free(s); return 0; }
int cudaStreamSynchronize(void *s) { return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { memcpy(d, s, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *st) { memset(d, v, n); return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int t, size_t b) { *n = 2; return 0; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t n, void *s) { return 0; }
int __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *n, void *s) {
  *n = 0;
  *(void **)s = 0;
  g->x = g->y = g->z = b->x = b->y = b->z = 1;
  return 0;
}
int cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t n, void *s) { return 0; }
int cudaFuncSetAttribute(const void *f, int a, int v) {
  attr[nattr].f = f;
  attr[nattr].dev = device;
  attr[nattr++].bytes = v;
  return 0;
}
int cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **a, size_t n, void *s) {
  int ok = n <= 48 * 1024, k;
  for (k = 0; k < nattr; k++)
    if (attr[k].f == f && attr[k].dev == device && (size_t)attr[k].bytes >= n) ok = 1;
  if (++launches == env("FAKE_REFUSE", 0)) return 999;
  return !ok ? 1 : (int)g.x > env("FAKE_SMS", 152) * (n > 114 * 1024 ? 1 : 4) ? 720 : 0;
}
