/* host_copy.cu -- see host_copy.h. */
#include "host_copy.h"

#include <algorithm>
#include <cstring>
#include <system_error>
#include <thread>

namespace oco {

bool host_pageable(const void *p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError(); /* an address the driver does not know */
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

void HostCopier::release() {
  for (auto &e : ev_) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  if (pinned_) cudaFreeHost(pinned_);
  pinned_ = nullptr;
  slot_ = 0;
}

cudaError_t HostCopier::ensure(size_t slot) {
  cudaError_t e = cudaSuccess;
  if (slot_ < slot) {
    release();
    e = cudaHostAlloc((void **)&pinned_, 2 * HOST_COPY_THREADS * slot, cudaHostAllocDefault);
    if (e == cudaSuccess) slot_ = slot;
  }
  for (auto &v : ev_)
    if (e == cudaSuccess && !v) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
  return e;
}

namespace {
/* Bytes [off, off + n) of the copies laid end to end, from the slot to their destinations. */
void scatter(const std::vector<HostCopy> &copies, size_t i, size_t off, const char *slot, size_t n) {
  const HostCopy &c = copies[i];
  while (n) {
    const size_t row = off / c.row_bytes, at = off - row * c.row_bytes, k = std::min(n, c.row_bytes - at);
    memcpy(c.dst + row * c.dst_pitch + at, slot, k);
    slot += k;
    off += k;
    n -= k;
  }
}

struct Piece {
  size_t copy, off, n;
};
}  // namespace

cudaError_t HostCopier::run(int device, cudaStream_t s, const std::vector<HostCopy> &copies) {
  cudaError_t e = cudaSuccess;
  size_t total = 0;
  for (const auto &c : copies) total += c.bytes();
  /* small outputs: one piece per thread, of at least a few pages */
  const size_t share = (total / HOST_COPY_THREADS + 4095) & ~(size_t)4095;
  const size_t size = std::min(slot_, std::max<size_t>(share, 64u << 10));
  std::vector<Piece> pieces;
  for (size_t i = 0; i < copies.size(); i++)
    for (size_t o = 0; o < copies[i].bytes(); o += size) pieces.push_back({i, o, std::min(size, copies[i].bytes() - o)});
  const int nt = (int)std::min<size_t>(HOST_COPY_THREADS, pieces.size());
  cudaError_t err[HOST_COPY_THREADS];
  std::fill(err, err + HOST_COPY_THREADS, cudaSuccess);
  auto work = [&](int t, int step) { /* pieces t, t + step, ... through the thread's two slots */
    cudaError_t q = cudaSetDevice(device);
    auto start = [&](size_t p, int b) {
      const Piece &x = pieces[p];
      char *slot = pinned_ + (2 * t + b) * slot_;
      q = cudaMemcpyAsync(slot, copies[x.copy].src + x.off, x.n, cudaMemcpyDeviceToHost, s);
      if (q == cudaSuccess) q = cudaEventRecord(ev_[2 * t + b], s);
    };
    int b = 0;
    if (q == cudaSuccess && (size_t)t < pieces.size()) start(t, 0);
    for (size_t p = t; q == cudaSuccess && p < pieces.size(); p += step, b ^= 1) {
      if (p + step < pieces.size()) start(p + step, b ^ 1);
      if (q == cudaSuccess) q = cudaEventSynchronize(ev_[2 * t + b]);
      if (q == cudaSuccess)
        scatter(copies, pieces[p].copy, pieces[p].off, pinned_ + (2 * t + b) * slot_, pieces[p].n);
    }
    err[t] = q;
  };
  std::thread th[HOST_COPY_THREADS];
  int made = 1;
  try {
    for (; made < nt; made++) th[made] = std::thread(work, made, nt);
  } catch (const std::system_error &) { /* fewer threads: this one takes the others' pieces below */
  }
  if (nt > 0) work(0, nt);
  for (int t = made; t < nt; t++) work(t, nt);
  for (int t = 1; t < made; t++) th[t].join();
  for (int t = 0; t < nt; t++)
    if (err[t] != cudaSuccess) e = err[t];
  if (e != cudaSuccess) cudaStreamSynchronize(s); /* nothing may still write the slots */
  return e;
}

}  // namespace oco
