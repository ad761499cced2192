/* A stand-in for the CUDA runtime on a machine without a GPU, preloaded ahead
 * of libcudart: device memory is host memory, kernels do nothing, and every
 * call that orders work is written to a journal (one line each: the call, its
 * stream, its event or copy direction), from which a test works out what waits
 * for what.  fake_fail_copy(k) makes the k-th copy from now on fail. */
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static char journal[1 << 20];
static size_t used;
static int fail_in;
static uintptr_t next_handle = 0x1000;
static struct { void *p; size_t n; } blocks[4096];
static int nblocks;

static void note(const char *op, const void *a, const void *b) {
  if (used + 128 < sizeof(journal))
    used += (size_t)snprintf(journal + used, 128, "%s %p %p\n", op, a, b);
}
const char *fake_journal(void) { return journal; }
void fake_clear(void) { used = 0; journal[0] = 0; }
void fake_fail_copy(int k) { fail_in = k; }
void fake_note(const char *op, void *stream) { note(op, stream, 0); }
/* start of the live device block of so many bytes (NULL: none, or several) */
void *fake_block(size_t bytes) {
  void *p = 0;
  for (int i = 0; i < nblocks; i++)
    if (blocks[i].n == bytes) {
      if (p) return 0;
      p = blocks[i].p;
    }
  return p;
}
static void *handle(void) { return (void *)(next_handle += 16); }

int cudaGetDeviceCount(int *n) { *n = 1; return 0; }
int cudaGetDevice(int *d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int *v, int attr, int dev) {
  *v = attr == 16 ? 148 : attr == 75 ? 10 : 0; /* SMs, compute capability 10.0 */
  (void)dev;
  return 0;
}
int cudaGetLastError(void) { return 0; }
int cudaPeekAtLastError(void) { return 0; }
int cudaFuncSetAttribute(const void *f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
static int encode_tiled() { return 0; }
int cudaGetDriverEntryPoint(const char *s, void **fn, unsigned long long fl, int *q) {
  (void)fl;
  *fn = strcmp(s, "cuTensorMapEncodeTiled") ? 0 : (void *)encode_tiled;
  if (q) *q = 0;
  return *fn ? 0 : 1;
}

int cudaMemPoolCreate(void **p, const void *pr) { (void)pr; *p = handle(); return 0; }
int cudaMemPoolSetAttribute(void *p, int a, void *v) { (void)p; (void)a; (void)v; return 0; }
int cudaDeviceSynchronize(void) { return 0; }
int cudaMemPoolTrimTo(void *p, size_t n) { (void)n; note("trim", p, 0); return 0; }
int cudaMallocFromPoolAsync(void **p, size_t n, void *pool, void *st) {
  (void)pool; (void)st;
  *p = calloc(1, n >> 32 ? 16 : n); /* (a block of 4 GiB and more is never touched) */
  blocks[nblocks].p = *p;
  blocks[nblocks++].n = n;
  return *p ? 0 : 2;
}
int cudaFreeAsync(void *p, void *st) {
  (void)st;
  for (int i = 0; i < nblocks; i++)
    if (blocks[i].p == p) {
      blocks[i] = blocks[--nblocks];
      break;
    }
  free(p);
  return 0;
}
int cudaMemsetAsync(void *p, int v, size_t n, void *st) {
  if (n <= 1 << 20) memset(p, v, n); /* (large blocks come zeroed and are never read) */
  note("memset", st, 0);
  return 0;
}
int cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st) {
  static const char *names[] = {"h2h", "h2d", "d2h", "d2d"};
  if (fail_in > 0 && --fail_in == 0) {
    note("failed", st, 0);
    return 1;
  }
  if (n <= 1 << 20) memcpy(d, s, n);
  note(kind >= 0 && kind < 4 ? names[kind] : "copy", st, kind == 2 ? d : s);
  return 0;
}

int cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; *s = handle(); return 0; }
int cudaStreamDestroy(void *s) { (void)s; return 0; }
int cudaStreamSynchronize(void *s) { note("sync", s, 0); return 0; }
int cudaEventCreate(void **e) { *e = handle(); return 0; }
int cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; *e = handle(); return 0; }
int cudaEventDestroy(void *e) { (void)e; return 0; }
int cudaEventRecord(void *e, void *s) { note("record", s, e); return 0; }
int cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)f; note("wait", s, e); return 0; }
int cudaLaunchKernelExC(const void *cfg, const void *f, void **args) {
  /* cudaLaunchConfig_t: two dim3 (24 bytes), the dynamic shared memory, the stream */
  void *st;
  (void)args;
  memcpy(&st, (const char *)cfg + 32, sizeof(st));
  note("kernel", st, f);
  return 0;
}
