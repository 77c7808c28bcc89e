// host_copy.cu on the host for tests/test_host_copy_host.py: the CUDA calls it makes are plain copies
// here, and operator new can fail from a given call on.
#include <cstdlib>
#include <cstring>
#include <new>

#include "host_copy.h"

static long g_allow = -1; // allocations before one fails (-1: none does)
void *operator new(size_t n) {
  if (g_allow == 0) throw std::bad_alloc();
  if (g_allow > 0) g_allow--;
  if (void *p = malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) { return cudaErrorInvalidValue; }
}

#include "host_copy.cu"

// Copies rows x row_bytes to rows dst_pitch apart, with the allocations after the first `allow` failing.
extern "C" int host_copy_run(const char *src, char *dst, size_t row_bytes, size_t dst_pitch, size_t rows, long allow) {
  oco::HostCopier c;
  const std::vector<oco::HostCopy> copies{{src, dst, row_bytes, dst_pitch, rows}};
  if (!c.ready(std::max(row_bytes * rows, oco::HOST_COPY_PIN))) return -1;
  g_allow = allow;
  const cudaError_t e = c.run(0, nullptr, copies);
  g_allow = -1;
  return (int)e;
}

// Whether each of n calls' outputs would go through the halves.
extern "C" void host_copy_ready(const size_t *bytes, int n, int *ready) {
  oco::HostCopier c;
  for (int i = 0; i < n; i++) ready[i] = c.ready(bytes[i]) ? 1 : 0;
}
