/* A stand-in for the CUDA runtime calls of a context and of ypdq_screen_host, preloaded on a
 * machine without a GPU. It keeps a list of what is allocated or created, fails the call it is
 * told to, and runs no kernel; copies to the host bring zeros. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

enum { kMax = 4096 };
static struct {
  void* p;
  char kind;
} live[kMax];
static int n_live, n_made, fail_at, attribute = 1 << 20, wrong_frees;
static char failed_kind;
static size_t most_pinned;

void fake_reset(int fail) { n_made = 0, fail_at = fail, failed_kind = 0, most_pinned = 0; }
void fake_attribute(int v) { attribute = v; }
int fake_live(void) { return n_live; }
int fake_made(void) { return n_made; }
int fake_wrong_frees(void) { return wrong_frees; }
int fake_failed_kind(void) { return failed_kind; }
size_t fake_most_pinned(void) { return most_pinned; }

static cudaError_t make(void** out, size_t bytes, char kind) {
  if (++n_made == fail_at || n_live == kMax) {
    failed_kind = kind;
    return cudaErrorMemoryAllocation;
  }
  *out = calloc(1, bytes ? bytes : 1);
  live[n_live].p = *out;
  live[n_live++].kind = kind;
  return cudaSuccess;
}
static cudaError_t drop(void* p, char kind) {
  for (int i = 0; i < n_live; ++i)
    if (live[i].p == p && live[i].kind == kind) {
      free(p);
      live[i] = live[--n_live];
      return cudaSuccess;
    }
  wrong_frees += p != NULL;
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return (void)d, cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount            ? 152
       : a == cudaDevAttrReservedSharedMemoryPerBlock ? 1024
                                                      : attribute;
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void* s, const void* p, size_t n, size_t o,
                               enum cudaMemcpyKind k) {
  return (void)s, (void)p, (void)n, (void)o, (void)k, cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  return (void)f, (void)a, (void)v, cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f) {
  (void)f;
  memset(a, 0, sizeof(*a));
  a->numRegs = 128;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int t,
                                                                   size_t s, unsigned flags) {
  return (void)f, (void)t, (void)s, (void)flags, *n = 0, cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) { return make(p, n > 4096 ? 4096 : n, 'd'); }
cudaError_t cudaFree(void* p) { return drop(p, 'd'); }
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (n > most_pinned) most_pinned = n;
  return make(p, n, 'h');
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) { return (void)f, make(p, n, 'h'); }
cudaError_t cudaFreeHost(void* p) { return drop(p, 'h'); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned f) {
  return (void)f, *d = h, cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  return (void)f, make((void**)s, 1, 's');
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s, 's'); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) {
  return (void)f, make((void**)e, 1, 'e');
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e, 'e'); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const struct cudaMemPoolProps* q) {
  return (void)q, make((void**)p, 1, 'p');
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void* v) {
  return (void)p, (void)a, (void)v, cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { return drop(p, 'p'); }

cudaError_t cudaStreamSynchronize(cudaStream_t s) { return (void)s, cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) {
  return (void)s, (void)e, (void)f, cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return (void)e, (void)s, cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  return (void)p, (void)v, (void)n, (void)s, cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, enum cudaMemcpyKind k,
                            cudaStream_t s) {
  (void)src, (void)s;
  if (k == cudaMemcpyDeviceToHost) memset(dst, 0, n);
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
  return (void)g, (void)b, (void)m, (void)s, 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  memset(g, 0, sizeof(*g));
  memset(b, 0, sizeof(*b));
  *m = 0;
  *(cudaStream_t*)s = NULL;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { return (void)f, *k = NULL, cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void** a, size_t m, cudaStream_t s) {
  return (void)k, (void)g, (void)b, (void)a, (void)m, (void)s, cudaSuccess;
}
