/* A stand-in for the CUDA runtime calls the library makes, for host-side tests without a GPU: device memory is host memory,
 * copies are memcpy, streams, events and graphs do nothing, and a kernel launch only tells the test (fake_on_launch) its name,
 * grid and arguments.  What the real runtime would refuse is refused: allocations beyond fake_memory bytes, and more than
 * 48 KB of dynamic shared memory on a device where the kernel's limit was not raised.  Preloaded by fake_runtime.py. */
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

enum { OK = 0, INVALID = 1, NO_MEMORY = 2 };
typedef struct { unsigned x, y, z; } dim3_;
typedef struct { dim3_ grid, block; size_t smem; void *stream, *attrs; unsigned n; } config;

size_t fake_memory = (size_t)1 << 40, fake_used, fake_peak;
int fake_device;
void (*fake_on_launch)(const char *name, const unsigned *grid, void **args);

static struct { const void *fn; const char *name; size_t smem[8]; } funcs[2048];
static int n_funcs, last_error;
static int ret(int e) { if (e) last_error = e; return e; }

void **__cudaRegisterFatBinary(void *p) { (void)p; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void) {}
void __cudaRegisterFunction(void **h, const void *fn, char *dev, const char *name) {
  (void)h; (void)dev;
  funcs[n_funcs].fn = fn;
  funcs[n_funcs++].name = name;
}
static __thread config pushed;
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t smem, void *st) {
  pushed = (config){g, b, smem, st, 0, 0};
  return 0;
}
int __cudaPopCallConfiguration(dim3_ *g, dim3_ *b, size_t *smem, void *st) {
  *g = pushed.grid; *b = pushed.block; *smem = pushed.smem; *(void **)st = pushed.stream;
  return OK;
}
static int at(const void *fn) { for (int i = 0; i < n_funcs; ++i) if (funcs[i].fn == fn) return i; return -1; }
static int launch(const void *fn, dim3_ g, size_t smem, void **args) {
  const int i = at(fn);
  if (i < 0 || (smem > 48 * 1024 && smem > funcs[i].smem[fake_device]))
    return ret(INVALID);
  if (fake_on_launch) fake_on_launch(funcs[i].name, &g.x, args);
  return OK;
}
int cudaLaunchKernel(const void *fn, dim3_ g, dim3_ b, void **args, size_t smem, void *st) {
  (void)b; (void)st;
  return launch(fn, g, smem, args);
}
int cudaLaunchKernelExC(const config *c, const void *fn, void **args) { return launch(fn, c->grid, c->smem, args); }
int cudaLaunchCooperativeKernel(const void *fn, dim3_ g, dim3_ b, void **args, size_t smem, void *st) {
  (void)b; (void)st;
  return launch(fn, g, smem, args);
}
int cudaFuncSetAttribute(const void *fn, int attr, int value) {
  const int i = at(fn);
  if (i < 0) return ret(INVALID);
  if (attr == 8) funcs[i].smem[fake_device] = (size_t)value;   /* cudaFuncAttributeMaxDynamicSharedMemorySize */
  return OK;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *fn, int t, size_t s, unsigned f) {
  (void)fn; (void)t; (void)s; (void)f; *n = 1; return OK;
}

/* the clusters of a B200 with 148 of its SMs in use; attribute 4 is the cluster's dimension */
int cudaOccupancyMaxActiveClusters(int *n, const void *fn, const config *c) {
  unsigned ctas = 1;
  for (unsigned i = 0; i < c->n; ++i)
    if (((const unsigned *)((const char *)c->attrs + 72 * i))[0] == 4) ctas = ((const unsigned *)((const char *)c->attrs + 72 * i))[2];
  if (at(fn) < 0 || funcs[at(fn)].smem[fake_device] < c->smem) return ret(INVALID);
  *n = ctas == 2 ? 74 : ctas == 4 ? 33 : ctas == 6 ? 22 : ctas == 8 ? 15 : 0;
  return *n ? OK : ret(INVALID);
}

int cudaGetDeviceCount(int *n) { *n = 8; return OK; }
int cudaGetDevice(int *d) { *d = fake_device; return OK; }
int cudaSetDevice(int d) { fake_device = d; return OK; }
int cudaDeviceGetAttribute(int *v, int a, int d) { (void)d; *v = a == 16 ? 148 : 1; return OK; }
int cudaDeviceSynchronize(void) { return OK; }
const char *cudaGetErrorString(int e) { return e == NO_MEMORY ? "out of memory" : e ? "invalid value" : "no error"; }
int cudaGetLastError(void) { int e = last_error; last_error = OK; return e; }
int cudaGetSymbolAddress(void **p, const void *s) { (void)s; *p = calloc(1, 2 << 20); return OK; }
static int entry(void) { return 0; }
int cudaGetDriverEntryPoint(const char *s, void **p, unsigned long long f, int *q) {
  (void)s; (void)f; *p = (void *)entry; if (q) *q = 0; return OK;
}

int cudaMalloc(void **p, size_t n) {
  *p = NULL;
  if (n > fake_memory || fake_used > fake_memory - n) return ret(NO_MEMORY);
  uint8_t *b = aligned_alloc(4096, (n + 8191) / 4096 * 4096);   /* a page in front holds the size */
  memset(b, 0, 4096);
  memset(b + 4096, 0, (n + 8191) / 4096 * 4096 - 4096);
  *(size_t *)b = n;
  fake_used += n;
  if (fake_used > fake_peak) fake_peak = fake_used;
  *p = b + 4096;
  return OK;
}
int cudaFree(void *p) {
  if (p) { uint8_t *b = (uint8_t *)p - 4096; fake_used -= *(size_t *)b; free(b); }
  return OK;
}
int cudaMallocAsync(void **p, size_t n, void *st) { (void)st; return cudaMalloc(p, n); }
int cudaFreeAsync(void *p, void *st) { (void)st; return cudaFree(p); }
int cudaMallocHost(void **p, size_t n) { *p = calloc(1, n ? n : 1); return OK; }
int cudaFreeHost(void *p) { free(p); return OK; }
int cudaHostRegister(void *p, size_t n, unsigned f) { (void)p; (void)n; (void)f; return OK; }
int cudaHostUnregister(void *p) { (void)p; return OK; }
int cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return OK; }
int cudaMemsetAsync(void *p, int v, size_t n, void *st) { (void)st; memset(p, v, n); return OK; }
int cudaMemcpy(void *d, const void *s, size_t n, int k) { (void)k; memmove(d, s, n); return OK; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { (void)k; (void)st; memmove(d, s, n); return OK; }
int cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, int k, void *st) {
  (void)k; (void)st;
  for (size_t i = 0; i < h; ++i) memmove((char *)d + i * dp, (const char *)s + i * sp, w);
  return OK;
}

static int handle(void **p) { static char h; *p = &h; return OK; }
int cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; return handle(s); }
int cudaStreamDestroy(void *s) { (void)s; return OK; }
int cudaStreamSynchronize(void *s) { (void)s; return OK; }
int cudaStreamBeginCapture(void *s, int m) { (void)s; (void)m; return OK; }
int cudaStreamEndCapture(void *s, void **g) { (void)s; return handle(g); }
int cudaGraphInstantiate(void **e, void *g, unsigned long long f) { (void)g; (void)f; return handle(e); }
int cudaGraphLaunch(void *e, void *s) { (void)e; (void)s; return OK; }
int cudaGraphDestroy(void *g) { (void)g; return OK; }
int cudaGraphExecDestroy(void *e) { (void)e; return OK; }
int cudaEventCreate(void **e) { return handle(e); }
int cudaEventDestroy(void *e) { (void)e; return OK; }
int cudaEventRecord(void *e, void *s) { (void)e; (void)s; return OK; }
int cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a; (void)b; *ms = 0.f; return OK; }
int cudaIpcGetMemHandle(void *h, void *p) { (void)h; (void)p; return ret(INVALID); }
int cudaIpcOpenMemHandle(void **p, ...) { *p = NULL; return ret(INVALID); }
int cudaIpcCloseMemHandle(void *p) { (void)p; return OK; }
