/* host_copy.cu -- see host_copy.h. */
#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
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
  half_ = 0;
}

cudaError_t HostCopier::ensure(size_t half) {
  cudaError_t e = cudaSuccess;
  if (half_ < half) {
    release();
    e = cudaHostAlloc((void **)&pinned_, 2 * half, cudaHostAllocDefault);
    if (e == cudaSuccess) half_ = half;
  }
  for (auto &v : ev_)
    if (e == cudaSuccess && !v) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
  return e;
}

namespace {
/* Calls f(copy, offset in it, n) for the parts of bytes [lo, hi) of the copies laid end to end. */
template <class F>
void parts(const std::vector<HostCopy> &copies, size_t lo, size_t hi, F f) {
  size_t at = 0;
  for (const auto &c : copies) {
    const size_t end = at + c.bytes();
    const size_t a = std::max(lo, at), b = std::min(hi, end);
    if (a < b) f(c, a - at, b - a);
    at = end;
  }
}

/* Bytes [lo, hi), which lie at slot, to their destinations. */
void scatter(const std::vector<HostCopy> &copies, size_t lo, size_t hi, const char *slot) {
  parts(copies, lo, hi, [&](const HostCopy &c, size_t off, size_t n) {
    while (n) {
      const size_t row = off / c.row_bytes, in = off - row * c.row_bytes, k = std::min(n, c.row_bytes - in);
      memcpy(c.dst + row * c.dst_pitch + in, slot, k);
      slot += k;
      off += k;
      n -= k;
    }
  });
}
}  // namespace

cudaError_t HostCopier::run(int device, cudaStream_t s, const std::vector<HostCopy> &copies) {
  (void)device; /* the calling thread's; the others do not talk to the driver */
  size_t total = 0;
  for (const auto &c : copies) total += c.bytes();
  const size_t rounds = (total + half_ - 1) / half_;
  const unsigned cores = std::thread::hardware_concurrency();
  const int nt = (int)std::max<size_t>(1, std::min<size_t>({(size_t)HOST_COPY_THREADS, total >> 19, cores / 2}));
  int made = 1;                     /* threads with a share, this one included */
  std::atomic<size_t> round{0};     /* rounds published; ~0: no more */
  std::atomic<int> left{0};         /* shares of the round still to be stored */
  auto share = [&](size_t r, int t, int n) { /* the t-th of n shares of round r */
    const size_t lo = r * half_, len = std::min(half_, total - lo);
    const size_t a = len * t / n, b = len * (t + 1) / n;
    scatter(copies, lo + a, lo + b, pinned_ + (r & 1) * half_ + a);
  };
  std::atomic<int> team{0}; /* = made once it is known */
  auto work = [&](int t) {
    for (size_t seen = 0;;) {
      size_t r;
      for (int spins = 0; (r = round.load(std::memory_order_acquire)) == seen;) {
        if (++spins < 4096) /* a round takes some 20 us; the first waits for the kernels */
          std::this_thread::yield();
        else
          std::this_thread::sleep_for(std::chrono::microseconds(50));
      }
      if (r == ~(size_t)0) return;
      share(r - 1, t, team.load(std::memory_order_relaxed));
      seen = r;
      left.fetch_sub(1, std::memory_order_release);
    }
  };
  auto start = [&](size_t r) { /* the DMA of round r into its half */
    const size_t lo = r * half_, hi = std::min(total, lo + half_);
    char *slot = pinned_ + (r & 1) * half_;
    cudaError_t e = cudaSuccess;
    parts(copies, lo, hi, [&](const HostCopy &c, size_t off, size_t n) {
      if (e == cudaSuccess) e = cudaMemcpyAsync(slot, c.src + off, n, cudaMemcpyDeviceToHost, s);
      slot += n;
    });
    return e == cudaSuccess ? cudaEventRecord(ev_[r & 1], s) : e;
  };
  cudaError_t e = rounds ? start(0) : cudaSuccess;
  std::thread th[HOST_COPY_THREADS];
  try {
    for (; made < nt; made++) th[made] = std::thread(work, made);
  } catch (...) { /* no thread or no memory for one: fewer threads, larger shares.  Nothing may leave here
                     past the started ones, which wait for a round */
  }
  team.store(made, std::memory_order_relaxed);
  for (size_t r = 0; r < rounds && e == cudaSuccess; r++) {
    if (r + 1 < rounds) e = start(r + 1); /* its half was stored in round r - 1 */
    if (e == cudaSuccess) e = cudaEventSynchronize(ev_[r & 1]);
    if (e != cudaSuccess) break;
    left.store(made - 1, std::memory_order_relaxed);
    round.store(r + 1, std::memory_order_release);
    share(r, 0, made);
    while (left.load(std::memory_order_acquire) > 0) std::this_thread::yield();
  }
  round.store(~(size_t)0, std::memory_order_release);
  for (int t = 1; t < made; t++) th[t].join();
  if (e != cudaSuccess) cudaStreamSynchronize(s); /* nothing may still write the halves */
  return e;
}

}  // namespace oco
