/* A CUDA runtime without a GPU, preloaded before libcudart by
 * tests/test_launch_pointers.py: two devices, memory from the host's heap that
 * is never reused, copies done at once, and launches reported to a callback
 * instead of run.  What libgbz hands to its kernels can then be looked at on
 * any machine. */
#define _GNU_SOURCE
#include <pthread.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

typedef int err;
enum { OK = 0, ENOMEM_ = 2, EINVAL_ = 1 };

/* ---- devices and allocations */
static __thread int device;
static __thread int copy_delay_us;
static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
struct alloc {
  char *p;
  uint64_t bytes;
  int device, freed;
  long filled; /* sequence number of the first completed cudaMemcpy into it */
};
static struct alloc *allocs;
static int nallocs, cap;
static long seq;

static struct alloc *find(const void *p) {
  for (int i = 0; i < nallocs; i++)
    if ((const char *)p >= allocs[i].p && (const char *)p < allocs[i].p + allocs[i].bytes) return &allocs[i];
  return 0;
}
/* 1 when p lies in a device allocation */
int fake_lookup(const void *p, int *dev, int *freed, long *filled, uint64_t *bytes) {
  pthread_mutex_lock(&mu);
  struct alloc *a = find(p);
  if (a) {
    *dev = a->device;
    *freed = a->freed;
    *filled = a->filled;
    *bytes = a->bytes;
  }
  pthread_mutex_unlock(&mu);
  return a != 0;
}
/* allocations that are not freed */
int fake_live(void) {
  int n = 0;
  pthread_mutex_lock(&mu);
  for (int i = 0; i < nallocs; i++) n += !allocs[i].freed;
  pthread_mutex_unlock(&mu);
  return n;
}
void fake_copy_delay(int us) { copy_delay_us = us; }

err cudaGetDevice(int *d) { *d = device; return OK; }
err cudaSetDevice(int d) { device = d; return d < 2 ? OK : EINVAL_; }
err cudaMalloc(void **p, size_t bytes) {
  *p = aligned_alloc(512, (bytes + 511) / 512 * 512);
  if (!*p) return ENOMEM_;
  memset(*p, 0, bytes);
  pthread_mutex_lock(&mu);
  if (nallocs == cap) allocs = realloc(allocs, sizeof(*allocs) * (cap = 2 * cap + 64));
  allocs[nallocs++] = (struct alloc){*p, bytes, device, 0, 0};
  pthread_mutex_unlock(&mu);
  return OK;
}
err cudaFree(void *p) {
  pthread_mutex_lock(&mu);
  struct alloc *a = p ? find(p) : 0;
  if (a) a->freed = 1;
  pthread_mutex_unlock(&mu);
  return !p || a ? OK : EINVAL_;
}
err cudaHostAlloc(void **p, size_t bytes, unsigned f) { (void)f; *p = calloc(1, bytes); return OK; }
err cudaFreeHost(void *p) { free(p); return OK; }
err cudaMemGetInfo(size_t *f, size_t *t) { *f = 200ull << 30; *t = 280ull << 30; return OK; }
err cudaMemcpy(void *d, const void *s, size_t n, int k) {
  (void)k;
  if (copy_delay_us) usleep(copy_delay_us);
  memcpy(d, s, n);
  pthread_mutex_lock(&mu);
  struct alloc *a = find(d);
  seq++;
  if (a && !a->filled) a->filled = seq;
  pthread_mutex_unlock(&mu);
  return OK;
}
err cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { (void)k; (void)st; memmove(d, s, n); return OK; }
err cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, int k, void *st) {
  (void)k;
  (void)st;
  for (size_t i = 0; i < h; i++) memmove((char *)d + i * dp, (const char *)s + i * sp, w);
  return OK;
}
err cudaMemsetAsync(void *d, int v, size_t n, void *st) { (void)st; memset(d, v, n); return OK; }

/* ---- streams, events, attributes */
static err handle(void **p) { *p = malloc(16); return OK; }
err cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; return handle(s); }
err cudaStreamCreateWithPriority(void **s, unsigned f, int p) { (void)f; (void)p; return handle(s); }
err cudaStreamDestroy(void *s) { (void)s; return OK; }
err cudaStreamSynchronize(void *s) { (void)s; return OK; }
err cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)s; (void)e; (void)f; return OK; }
err cudaStreamQuery(void *s) { (void)s; return OK; }
err cudaEventCreate(void **e) { return handle(e); }
err cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; return handle(e); }
err cudaEventDestroy(void *e) { (void)e; return OK; }
err cudaEventRecord(void *e, void *s) { (void)e; (void)s; return OK; }
err cudaEventQuery(void *e) { (void)e; return OK; }
err cudaEventSynchronize(void *e) { (void)e; return OK; }
err cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a; (void)b; *ms = 1; return OK; }
err cudaDeviceSynchronize(void) { return OK; }
err cudaDeviceGetAttribute(int *v, int a, int d) { (void)a; (void)d; *v = 152; return OK; }
err cudaDeviceGetStreamPriorityRange(int *a, int *b) { *a = 0; *b = -1; return OK; }
err cudaFuncSetAttribute(const void *f, int a, int v) { (void)f; (void)a; (void)v; return OK; }
err cudaGetLastError(void) { return OK; }

/* ---- kernels */
static struct { const void *fn; const char *name; } kernels[4096];
static int nkernels;
void __cudaRegisterFunction(void **h, const char *fn, char *dfn, const char *name, int lim, void *t, void *b, void *bd,
                            void *gd, int *ws) {
  (void)h, (void)dfn, (void)lim, (void)t, (void)b, (void)bd, (void)gd, (void)ws;
  if (nkernels < 4096) {
    kernels[nkernels].fn = fn;
    kernels[nkernels++].name = name;
  }
}
typedef void (*launch_cb)(const char *name, int device, long seq, void **args);
static launch_cb on_launch;
void fake_on_launch(launch_cb cb) { on_launch = cb; }
err cudaLaunchKernelExC(const void *cfg, const void *fn, void **args) {
  (void)cfg;
  pthread_mutex_lock(&mu);
  const long at = ++seq;
  pthread_mutex_unlock(&mu);
  for (int i = 0; on_launch && i < nkernels; i++)
    if (kernels[i].fn == fn) {
      on_launch(kernels[i].name, device, at, args);
      break;
    }
  return OK;
}
