/* A CUDA runtime without a GPU, preloaded by the tests of the library's host
 * code (fake_runtime.py): device memory is host memory, launches do nothing
 * but check what a launch checks on the host, and a test can make calls fail.
 * Streams, events and pools are handles without a meaning. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#define API __attribute__((visibility("default")))

/* ---- what a test sets and reads */
API int fake_fail_launch = -1;                  /* launches until one fails; < 0: none does */
API long long fake_pool_limit = -1;             /* most bytes of pool allocations; < 0: any */
API long long fake_pool_live = 0;               /* bytes of them not freed */
API long long fake_launches = 0;
API long long fake_malloc_live = 0;             /* cudaMalloc'ed pieces not freed */
API long long fake_capture = 0;                 /* id of a capture in progress; 0: none */
API void (*fake_attribute_set)(void) = NULL;    /* called after a kernel's attribute is set */

static cudaError_t last = cudaSuccess;
static cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}

/* ---- launches: the shared memory asked for is within the kernel's limit */
static struct {
  const void *f;
  size_t smem;
} limit[256];
static int nlimit = 0;

static cudaError_t launch(const void *f, size_t smem) {
  size_t most = 48 * 1024;
  for (int i = 0; i < nlimit; i++)
    if (limit[i].f == f) most = limit[i].smem;
  fake_launches++;
  if (smem > most) return done(cudaErrorInvalidValue);
  if (fake_fail_launch >= 0 && fake_fail_launch-- == 0) return done(cudaErrorLaunchOutOfResources);
  return cudaSuccess;
}
API cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int value) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  if (value < 0 || value > 227 * 1024) return done(cudaErrorInvalidValue);
  int i = 0;
  while (i < nlimit && limit[i].f != f) i++;
  if (i == nlimit) nlimit++;
  limit[i].f = f;
  limit[i].smem = (size_t)value;
  if (fake_attribute_set) fake_attribute_set();
  return cudaSuccess;
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  (void)args;
  return launch(f, c->dynamicSmemBytes);
}
API cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
API cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void **args, size_t smem,
                                   cudaStream_t st) {
  (void)grid, (void)block, (void)args, (void)st;
  return launch((const void *)k, smem);
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int t,
                                                                       size_t smem, unsigned fl) {
  (void)f, (void)t, (void)smem, (void)fl;
  *n = 1;
  return cudaSuccess;
}

/* ---- memory */
API cudaError_t cudaMalloc(void **p, size_t n) {
  *p = calloc(n ? n : 1, 1);
  fake_malloc_live++;
  return *p ? cudaSuccess : done(cudaErrorMemoryAllocation);
}
API cudaError_t cudaHostAlloc(void **p, size_t n, unsigned flags) {
  (void)flags;
  return cudaMalloc(p, n);
}
API cudaError_t cudaFree(void *p) {
  fake_malloc_live -= p != NULL;
  free(p);
  return cudaSuccess;
}
API cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
API cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) {
  (void)k;
  memcpy(d, s, n);
  return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k,
                                cudaStream_t st) {
  (void)st;
  return cudaMemcpy(d, s, n, k);
}
API cudaError_t cudaMemset(void *d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
API cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  (void)st;
  return cudaMemset(d, v, n);
}
API cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
  (void)p;
  memset(a, 0, sizeof *a);
  return cudaSuccess;
}

/* ---- pools: an allocation carries its size in front */
API cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const struct cudaMemPoolProps *props) {
  (void)props;
  *p = (cudaMemPool_t)malloc(1);
  return cudaSuccess;
}
API cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
  free(p);
  return cudaSuccess;
}
API cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void *v) {
  (void)p, (void)a, (void)v;
  return cudaSuccess;
}
API cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t pool, cudaStream_t st) {
  (void)pool, (void)st;
  if (fake_pool_limit >= 0 && fake_pool_live + (long long)n > fake_pool_limit)
    return done(cudaErrorMemoryAllocation);
  char *q = malloc(n + 64);
  memcpy(q, &n, sizeof n);
  fake_pool_live += (long long)n;
  *p = q + 64;
  return cudaSuccess;
}
API cudaError_t cudaFreeAsync(void *p, cudaStream_t st) {
  (void)st;
  size_t n;
  memcpy(&n, (char *)p - 64, sizeof n);
  fake_pool_live -= (long long)n;
  free((char *)p - 64);
  return cudaSuccess;
}

/* ---- captures: what the graph holds is let go by fake_graph_gone */
static struct {
  cudaHostFn_t f;
  void *p;
} held[64];
static int nheld = 0;

API cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, enum cudaStreamCaptureStatus *st,
                                         unsigned long long *id, cudaGraph_t *g,
                                         const cudaGraphNode_t **d, const cudaGraphEdgeData **e,
                                         size_t *n) {
  (void)s, (void)d, (void)e, (void)n;
  *st = fake_capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  if (id) *id = (unsigned long long)fake_capture;
  if (g) *g = (cudaGraph_t)&held;
  return cudaSuccess;
}
API cudaError_t cudaThreadExchangeStreamCaptureMode(enum cudaStreamCaptureMode *m) {
  (void)m;
  return cudaSuccess;
}
API cudaError_t cudaUserObjectCreate(cudaUserObject_t *o, void *p, cudaHostFn_t f, unsigned count,
                                     unsigned flags) {
  (void)count, (void)flags;
  held[nheld].f = f;
  held[nheld].p = p;
  *o = (cudaUserObject_t)&held[nheld++];
  return cudaSuccess;
}
API cudaError_t cudaGraphRetainUserObject(cudaGraph_t g, cudaUserObject_t o, unsigned count,
                                          unsigned flags) {
  (void)g, (void)o, (void)count, (void)flags;
  return cudaSuccess;
}
API cudaError_t cudaUserObjectRelease(cudaUserObject_t o, unsigned count) {
  (void)o, (void)count;
  return cudaSuccess;
}
API void fake_graph_gone(void) {
  while (nheld > 0) {
    nheld--;
    held[nheld].f(held[nheld].p);
  }
}

/* ---- device, streams, events, errors */
API cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
API cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) {
  (void)f;
  *s = (cudaStream_t)malloc(1);
  return cudaSuccess;
}
API cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
API cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  (void)s;
  return cudaSuccess;
}
API cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) {
  (void)s, (void)e, (void)f;
  return cudaSuccess;
}
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) {
  (void)f;
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
API cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
API cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  (void)e, (void)s;
  return cudaSuccess;
}
API cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  (void)e;
  return cudaSuccess;
}
API cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
