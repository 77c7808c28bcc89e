/*
 * host_copy.h -- device -> pageable host copies of the host-array block solve.
 *
 * The driver's copy into pageable memory runs at ~15 GB/s on one thread and takes the page faults
 * of a fresh array on the way (the reference deck's 31 x 32 x 33 block with 5 wavelengths, 4.2 MB of
 * outputs into new arrays: 1.43 ms a call of which the GPU works 0.11 ms).  Here up to
 * HOST_COPY_THREADS threads take turns on the pieces of the outputs, each with two pinned slots of
 * its own: the next piece's DMA is in flight while the thread stores the current one, and the
 * faults of different pieces overlap: 0.72 ms a call.  Pinned arrays of the caller are copied into
 * directly.
 */
#ifndef OCO_HOST_COPY_H
#define OCO_HOST_COPY_H

#include <cstddef>
#include <vector>

#include <cuda_runtime.h>

namespace oco {

constexpr int HOST_COPY_THREADS = 8;
/* Bytes per pinned slot: 2 MB in all (pinning 8 MB takes 8 ms of a context's first call), 16 MB for
 * outputs of HOST_COPY_LARGE and more. */
constexpr size_t HOST_COPY_PIECE = 128u << 10, HOST_COPY_PIECE_LARGE = 1u << 20;
constexpr size_t HOST_COPY_LARGE = 64u << 20;
constexpr size_t HOST_COPY_MIN = 512u << 10;   /* smaller outputs take the driver's copies */

/* rows x row_bytes, contiguous at src (device), dst_pitch bytes apart at dst (host). */
struct HostCopy {
  const char *src;
  char *dst;
  size_t row_bytes, dst_pitch, rows;
  size_t bytes() const { return row_bytes * rows; }
};

/* The pinned slots and events of one context (one call at a time, as the context's staging). */
class HostCopier {
 public:
  ~HostCopier() { release(); }
  /* Allocates the slots for outputs of `bytes` (false: no memory for them; the driver's copies do
   * without). */
  bool ready(size_t bytes) {
    if (ensure(bytes >= HOST_COPY_LARGE ? HOST_COPY_PIECE_LARGE : HOST_COPY_PIECE) == cudaSuccess) return true;
    cudaGetLastError();
    release();
    return false;
  }
  /* Copies all (after ready()), after the work enqueued on s so far; returns when the host arrays are complete. */
  cudaError_t run(int device, cudaStream_t s, const std::vector<HostCopy> &copies);
  void release();

 private:
  cudaError_t ensure(size_t slot);
  char *pinned_ = nullptr;
  size_t slot_ = 0; /* bytes per slot */
  cudaEvent_t ev_[2 * HOST_COPY_THREADS] = {};
};

/* Whether p is ordinary (pageable) host memory. */
bool host_pageable(const void *p);

}  // namespace oco

#endif /* OCO_HOST_COPY_H */
