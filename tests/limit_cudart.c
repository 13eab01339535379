/* Preloaded into a child process: device allocations pass through to the CUDA
 * runtime, except that after limit_exact(bytes, n) every allocation of exactly
 * `bytes` beyond the first n of them fails as if the device were full. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

#include <cuda_runtime_api.h>

static size_t size;
static long left;
static unsigned long refused;

void limit_exact(size_t bytes, long n) { size = bytes; left = n; }
void limit_off(void) { size = 0; }
unsigned long limit_refused(void) { return refused; }

cudaError_t cudaMalloc(void **p, size_t n) {
  static cudaError_t (*real)(void **, size_t);
  if (!real) {
    void *rt = dlopen("libcudart.so.13", RTLD_NOLOAD | RTLD_LAZY);
    real = rt ? (cudaError_t(*)(void **, size_t))dlsym(rt, "cudaMalloc") : NULL;
    if (!real) return cudaErrorUnknown;
  }
  if (size && n == size && left-- <= 0) {
    refused++;
    return cudaErrorMemoryAllocation;
  }
  return real(p, n);
}
