/* Preloaded over the CUDA runtime: allocations from a memory pool of more than
 * POOL_LIMIT bytes (environment) fail as they do when the device is full. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stdlib.h>

typedef cudaError_t (*alloc_fn)(void **, size_t, cudaMemPool_t, cudaStream_t);

__attribute__((visibility("default"))) cudaError_t cudaMallocFromPoolAsync(void **p, size_t n,
                                                                           cudaMemPool_t pool,
                                                                           cudaStream_t st) {
  const char *limit = getenv("POOL_LIMIT");
  if (limit && n > strtoull(limit, NULL, 10)) return cudaErrorMemoryAllocation;
  /* the runtime that the library has loaded */
  void *rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
  alloc_fn f = rt ? (alloc_fn)dlsym(rt, "cudaMallocFromPoolAsync") : NULL;
  return f ? f(p, n, pool, st) : cudaErrorInitializationError;
}
