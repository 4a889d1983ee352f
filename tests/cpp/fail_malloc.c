/* Preloaded by tests/test_gpu_allocation_failures.py, which hands it the
 * runtime's own cudaMalloc: the n-th call after fail_malloc_at(n) asks for more
 * memory than any device has, so that the runtime reports it out of memory. */
#include <stddef.h>

typedef int (*malloc_fn)(void **, size_t);

static malloc_fn real;
static long left;

void fail_malloc_real(void *f) { real = (malloc_fn)f; }
void fail_malloc_at(long n) { left = n; }

int cudaMalloc(void **p, size_t bytes) {
  if (left > 0 && --left == 0) bytes = (size_t)1 << 60;
  return real(p, bytes);
}
