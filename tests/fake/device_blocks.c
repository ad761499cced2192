/* Preloaded ahead of libcudart, on a machine with a GPU: notes where the library's
 * blocks of device memory lie, and passes every call on. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

static struct { void *p; size_t n; } blocks[4096];
static int nblocks;

static void *real(const char *name) {
  static void *lib;
  if (!lib) lib = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  return lib ? dlsym(lib, name) : 0;
}
int cudaMallocFromPoolAsync(void **p, size_t n, void *pool, void *st) {
  int (*f)(void **, size_t, void *, void *) = (int (*)(void **, size_t, void *, void *))real("cudaMallocFromPoolAsync");
  int rc = f ? f(p, n, pool, st) : 35;
  if (!rc && nblocks < 4096) {
    blocks[nblocks].p = *p;
    blocks[nblocks++].n = n;
  }
  return rc;
}
/* the block of so many bytes taken last */
void *block_of(size_t bytes) {
  for (int i = nblocks - 1; i >= 0; i--)
    if (blocks[i].n == bytes) return blocks[i].p;
  return 0;
}
