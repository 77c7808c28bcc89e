/*
 * host_copy.h -- device -> pageable host copies of the host-array block solve.
 *
 * The driver's copy into pageable memory runs at ~15 GB/s on one thread and takes the page faults
 * of a fresh array on the way (the reference deck's 31 x 32 x 33 block with 5 wavelengths, 4.2 MB of
 * outputs into new arrays: 1.43 ms a call of which the GPU works 0.11 ms).  Here the outputs pass
 * through two pinned halves: while one fills by DMA, up to HOST_COPY_THREADS threads store the other
 * and take its faults together: 0.70 ms a call (14 MB of outputs 1.19 -> 0.86 ms, 157 MB 38 -> 12
 * ms).  One thread alone talks to the driver: eight with slots of their own spent more on its lock
 * than the copies took (14 MB: 1.23 ms).  Pinned arrays of the caller are copied into directly.
 */
#ifndef OCO_HOST_COPY_H
#define OCO_HOST_COPY_H

#include <cstddef>
#include <vector>

#include <cuda_runtime.h>

namespace oco {

constexpr int HOST_COPY_THREADS = 8;
constexpr size_t HOST_COPY_MIN = 512u << 10; /* smaller outputs take the driver's copies */
/* Bytes of a pinned half: 2 MB in all (pinning 8 MB takes 8 ms of a context's first call), 16 MB for
 * outputs of HOST_COPY_LARGE and more. */
constexpr size_t HOST_COPY_HALF = 1u << 20, HOST_COPY_HALF_LARGE = 8u << 20;
constexpr size_t HOST_COPY_LARGE = 64u << 20;

/* rows x row_bytes, contiguous at src (device), dst_pitch bytes apart at dst (host). */
struct HostCopy {
  const char *src;
  char *dst;
  size_t row_bytes, dst_pitch, rows;
  size_t bytes() const { return row_bytes * rows; }
};

/* The pinned halves and events of one context (one call at a time, as the context's staging). */
class HostCopier {
 public:
  ~HostCopier() { release(); }
  /* Allocates the halves for outputs of `bytes` (false: no memory for them; the driver's copies do
   * without). */
  bool ready(size_t bytes) {
    if (ensure(bytes >= HOST_COPY_LARGE ? HOST_COPY_HALF_LARGE : HOST_COPY_HALF) == cudaSuccess) return true;
    cudaGetLastError();
    release();
    return false;
  }
  /* Copies all (after ready()), after the work enqueued on s so far; returns when the host arrays are complete. */
  cudaError_t run(int device, cudaStream_t s, const std::vector<HostCopy> &copies);
  void release();

 private:
  cudaError_t ensure(size_t half);
  char *pinned_ = nullptr;
  size_t half_ = 0; /* bytes per half */
  cudaEvent_t ev_[2] = {};
};

/* Whether p is ordinary (pageable) host memory. */
bool host_pageable(const void *p);

}  // namespace oco

#endif /* OCO_HOST_COPY_H */
