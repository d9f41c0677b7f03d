/* fake_cudart.c -- a CUDA runtime without a GPU, for tests of the library's host code:
 * preloaded in a child process (tests/fakecuda.py), it hands out addresses that are
 * never touched, runs no kernel, copies nothing, and logs every call that allocates,
 * frees, enqueues or waits, one line each, to the file FAKE_LOG names.
 *   FAKE_MEMORY  bytes of the device: an allocation past them fails
 *   FAKE_FAIL    part of a kernel's name: its first launch returns an error
 *   FAKE_COPIES, FAKE_COPY_BYTES  a file to append the host data of copies of so many
 *                bytes to
 * Device-to-host copies leave their target as it is (pinned memory starts at zero: no
 * error, no change), so a solve ends after its first sweeps. */
#define _GNU_SOURCE
#include <pthread.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define BASE 0x500000000000ull /* device addresses: [BASE, BASE + 2^42) */

static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static FILE *out;
static uint64_t next_ptr = BASE, used, limit = 1ull << 38;
static int next_id = 1, last_error, failed;
/* the primary context: its id, and the first stream and address made in it */
static unsigned long long ctx_id = 1;
static int first_stream = 1;
static uint64_t first_ptr = BASE;
static struct { uint64_t p, n; } blocks[4096];
static int nblocks;
static struct { const void *fn; char name[256]; } kernels[4096];
static int nkernels;

__attribute__((constructor)) static void init(void) {
  const char *f = getenv("FAKE_LOG"), *m = getenv("FAKE_MEMORY");
  out = f ? fopen(f, "w") : NULL;
  if (m) limit = strtoull(m, NULL, 0);
}
#define SAY(...) (out ? (fprintf(out, __VA_ARGS__), fflush(out)) : 0)

typedef struct { unsigned x, y, z; } dim3_;

/* A stream or an address of a context that a reset ended: logged, and an error. */
static int stale(const void *st, const void *p) {
  const int s = (int)(intptr_t)st;
  const uint64_t q = (uint64_t)(uintptr_t)p;
  const int bad = (s && s < first_stream) || (q >= BASE && q < first_ptr);
  if (bad) SAY("stale stream%d %llx\n", s, (unsigned long long)q);
  return bad ? (last_error = 400) : 0; /* cudaErrorInvalidResourceHandle */
}
int cudaDeviceReset(void) {
  SAY("reset\n");
  ++ctx_id;
  first_stream = next_id;
  first_ptr = next_ptr;
  used = 0;
  nblocks = 0;
  return 0;
}

/* launches */
void **__cudaRegisterFatBinary(void *p) { return (void **)p; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *a, char *b, const char *c, int d, size_t e, int f, int g) {
  (void)h; (void)a; (void)b; (void)c; (void)d; (void)e; (void)f; (void)g;
}
void __cudaRegisterFunction(void **h, const char *fn, char *df, const char *name, int lim, void *t, void *b, void *bd,
                            void *gd, int *ws) {
  (void)h; (void)df; (void)lim; (void)t; (void)b; (void)bd; (void)gd; (void)ws;
  if (nkernels < 4096) {
    kernels[nkernels].fn = fn;
    snprintf(kernels[nkernels++].name, 256, "%s", name);
  }
}
int __cudaGetKernel(void **k, const void *fn) {
  *k = (void *)fn;
  return 0;
}
static __thread dim3_ cfg_g, cfg_b;
static __thread size_t cfg_s;
static __thread void *cfg_st;
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t s, void *st) {
  cfg_g = g;
  cfg_b = b;
  cfg_s = s;
  cfg_st = st;
  return 0;
}
int __cudaPopCallConfiguration(dim3_ *g, dim3_ *b, size_t *s, void *st) {
  *g = cfg_g;
  *b = cfg_b;
  *s = cfg_s;
  *(void **)st = cfg_st;
  return 0;
}
int __cudaLaunchKernel(void *k, dim3_ g, dim3_ b, void **args, size_t s, void *st) {
  (void)b; (void)args; (void)s;
  if (stale(st, NULL)) return 400;
  const char *name = "?", *f = getenv("FAKE_FAIL");
  pthread_mutex_lock(&mu);
  for (int i = 0; i < nkernels; ++i)
    if (kernels[i].fn == k) name = kernels[i].name;
  const int bad = f && !failed && strstr(name, f);
  if (bad) {
    failed = 1;
    last_error = 719; /* cudaErrorLaunchFailure */
  }
  SAY("%s %s %u stream%d\n", bad ? "fail" : "launch", name, g.x, (int)(intptr_t)st);
  pthread_mutex_unlock(&mu);
  return bad ? last_error : 0;
}

/* memory */
int cudaMalloc(void **p, size_t n) {
  pthread_mutex_lock(&mu);
  int e = 0;
  if (used + n > limit || nblocks == 4096) {
    e = last_error = 2; /* cudaErrorMemoryAllocation */
    SAY("nomem %zu\n", n);
  } else {
    used += n;
    blocks[nblocks].p = next_ptr;
    blocks[nblocks++].n = n;
    *p = (void *)next_ptr;
    next_ptr += (n + 511) & ~511ull;
    SAY("malloc %zu\n", n);
  }
  pthread_mutex_unlock(&mu);
  return e;
}
int cudaFree(void *p) {
  if (stale(NULL, p)) return 400;
  pthread_mutex_lock(&mu);
  for (int i = 0; i < nblocks; ++i)
    if (p && blocks[i].p == (uint64_t)(uintptr_t)p) {
      used -= blocks[i].n;
      SAY("free %zu\n", (size_t)blocks[i].n);
      blocks[i] = blocks[--nblocks];
      break;
    }
  pthread_mutex_unlock(&mu);
  return 0;
}
int cudaHostAlloc(void **p, size_t n, unsigned f) {
  (void)f;
  *p = calloc(1, n);
  return *p ? 0 : 2;
}
int cudaFreeHost(void *p) {
  free(p);
  return 0;
}
int cudaMemGetInfo(size_t *fr, size_t *tot) {
  *fr = limit - used;
  *tot = limit;
  return 0;
}
struct attrs { int type, device; void *dp, *hp; long reserved[8]; };
int cudaPointerGetAttributes(struct attrs *a, const void *p) {
  const uint64_t q = (uint64_t)(uintptr_t)p;
  memset(a, 0, 4 * sizeof(void *) - 8);
  a->type = q >= BASE && q < BASE + (1ull << 42) ? 2 : 0; /* device, unregistered */
  return 0;
}
int cudaMemcpy(void *d, const void *s, size_t n, int k) {
  (void)d; (void)s; (void)k;
  SAY("copy %zu stream0\n", n);
  return 0;
}
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) {
  (void)k;
  if (stale(st, d) || stale(st, s)) return 400;
  const char *f = getenv("FAKE_COPIES"), *b = getenv("FAKE_COPY_BYTES");
  if (f && b && (size_t)atoll(b) == n && (uint64_t)(uintptr_t)s < BASE) {
    FILE *o = fopen(f, "ab");
    fwrite(s, 1, n, o);
    fclose(o);
  }
  SAY("copy %zu stream%d\n", n, (int)(intptr_t)st);
  return 0;
}
int cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, int k, void *st) {
  (void)d; (void)dp; (void)s; (void)sp; (void)k;
  SAY("copy %zu stream%d\n", w * h, (int)(intptr_t)st);
  return 0;
}
int cudaMemset(void *d, int v, size_t n) {
  (void)d; (void)v;
  SAY("set %zu stream0\n", n);
  return 0;
}
int cudaMemsetAsync(void *d, int v, size_t n, void *st) {
  (void)v;
  if (stale(st, d)) return 400;
  SAY("set %zu stream%d\n", n, (int)(intptr_t)st);
  return 0;
}

/* streams, events, graphs */
int cudaStreamCreateWithFlags(void **s, unsigned f) {
  (void)f;
  *s = (void *)(intptr_t)__sync_fetch_and_add(&next_id, 1);
  return 0;
}
int cudaStreamDestroy(void *s) {
  if (stale(s, NULL)) return 400;
  SAY("destroy stream%d\n", (int)(intptr_t)s);
  return 0;
}
int cudaStreamSynchronize(void *s) {
  if (stale(s, NULL)) return 400;
  SAY("wait stream%d\n", (int)(intptr_t)s);
  return 0;
}
int cudaStreamWaitEvent(void *s, void *e, unsigned f) {
  (void)s; (void)e; (void)f;
  return 0;
}
int cudaDeviceSynchronize(void) { return 0; }
int cudaEventCreate(void **e) {
  *e = (void *)1;
  return 0;
}
int cudaEventCreateWithFlags(void **e, unsigned f) {
  (void)f;
  *e = (void *)1;
  return 0;
}
int cudaEventDestroy(void *e) {
  (void)e;
  return 0;
}
int cudaEventRecord(void *e, void *s) {
  (void)e; (void)s;
  return 0;
}
int cudaEventSynchronize(void *e) {
  (void)e;
  return 0;
}
int cudaEventElapsedTime(float *ms, void *a, void *b) {
  (void)a; (void)b;
  *ms = 0.0f;
  return 0;
}
int cudaStreamBeginCapture(void *s, int m) {
  (void)s; (void)m;
  return 0;
}
int cudaStreamEndCapture(void *s, void **g) {
  (void)s;
  *g = (void *)1;
  return 0;
}
int cudaGraphInstantiate(void **x, void *g, unsigned long long f) {
  (void)g; (void)f;
  *x = (void *)1;
  return 0;
}
int cudaGraphLaunch(void *x, void *s) {
  (void)x; (void)s;
  return 0;
}
int cudaGraphDestroy(void *g) {
  (void)g;
  return 0;
}
int cudaGraphExecDestroy(void *x) {
  (void)x;
  return 0;
}

/* device */
int cudaGetDeviceCount(int *n) {
  *n = 1;
  return 0;
}
int cudaGetDevice(int *d) {
  *d = 0;
  return 0;
}
int cudaSetDevice(int d) {
  (void)d;
  return 0;
}
int cudaDeviceGetAttribute(int *v, int a, int d) {
  (void)a; (void)d;
  *v = 152;
  return 0;
}
int cudaFuncSetAttribute(const void *f, int a, int v) {
  (void)f; (void)a; (void)v;
  return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl) {
  (void)f; (void)b; (void)s; (void)fl;
  *n = 1;
  return 0;
}
int cudaGetSymbolAddress(void **p, const void *s) {
  (void)s;
  *p = (void *)BASE;
  return 0;
}
static int encode_ok(void) { return 0; }
static int get_current(void **c) {
  *c = (void *)1;
  return 0;
}
static int get_id(void *c, unsigned long long *id) {
  (void)c;
  *id = ctx_id;
  return 0;
}
int cudaGetDriverEntryPointByVersion(const char *n, void **p, unsigned v, unsigned long long f, int *q) {
  (void)v; (void)f;
  *p = !strcmp(n, "cuCtxGetCurrent") ? (void *)get_current : !strcmp(n, "cuCtxGetId") ? (void *)get_id : (void *)encode_ok;
  if (q) *q = 0;
  return 0;
}
int cudaGetLastError(void) {
  const int e = last_error;
  last_error = 0;
  return e;
}
const char *cudaGetErrorString(int e) {
  (void)e;
  return "fake error";
}
