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
/* Smaller outputs take the driver's copies: starting the threads costs a call some 0.1 ms, which arrays that
 * the caller keeps (no faults) never give back (kept / fresh arrays, driver's copies and these: 2 MB 0.35
 * and 0.61 ms / 1.21 and 0.84 ms; 3 MB 0.43 and 0.45 / 1.71 and 0.80; 3.5 MB 0.47 and 0.38 / 1.98 and
 * 0.86). */
constexpr size_t HOST_COPY_MIN = 3u << 20;
/* Output bytes that a context has seen when it pins its halves, which takes 1.5-2 ms of that call (4 MB: 4.6
 * -> 6.5 ms for a context's first call): a process that solves one small block is better off without,
 * 8 MB break even in one call (7.2 ms both). */
constexpr size_t HOST_COPY_PIN = 8u << 20;
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
  /* Whether outputs of `bytes` go through the halves: once the context's calls have brought HOST_COPY_PIN,
   * and there is memory for them; otherwise the driver's copies do. */
  bool ready(size_t bytes) {
    if (bytes < HOST_COPY_MIN) return false;
    seen_ += bytes;
    if (seen_ < HOST_COPY_PIN) return false;
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
  size_t seen_ = 0; /* output bytes of the calls so far that could have used the halves */
  cudaEvent_t ev_[2] = {};
};

/* Whether p is ordinary (pageable) host memory. */
bool host_pageable(const void *p);

}  // namespace oco

#endif /* OCO_HOST_COPY_H */
