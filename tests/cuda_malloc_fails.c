/* Preloaded: the k-th cudaMalloc after malloc_fails_at(k) reports that the
 * device is out of memory; malloc_calls() counts them. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

static long calls, fail_at;
void malloc_fails_at(long k) { calls = 0; fail_at = k; }
long malloc_calls(void) { return calls; }

int cudaMalloc(void** p, size_t n) {
  static int (*real)(void**, size_t);
  if (!real) {
    void* lib = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    if (lib) real = (int (*)(void**, size_t))dlsym(lib, "cudaMalloc");
    if (!real) return 35;
  }
  ++calls;
  if (calls == fail_at) return 2; /* cudaErrorMemoryAllocation */
  return real(p, n);
}
