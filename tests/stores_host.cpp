// Host build of stores.h for tests/test_stores_host.py: 32 threads stand in for the lanes of a warp.
#include <pthread.h>
#include <unistd.h>

#include <atomic>
#include <cstdint>
#include <thread>
#include <vector>

struct Idx {
  unsigned x;
};
static thread_local Idx threadIdx;
static pthread_barrier_t g_warp;
static unsigned long long g_exchange[32];

static void __syncwarp() { pthread_barrier_wait(&g_warp); }
template <class T>
static T __shfl_sync(unsigned, T v, int src) {
  g_exchange[threadIdx.x] = (unsigned long long)v;
  __syncwarp();
  const T r = (T)g_exchange[src];
  __syncwarp();
  return r;
}
static unsigned __ballot_sync(unsigned, bool on) {
  g_exchange[threadIdx.x] = on;
  __syncwarp();
  unsigned m = 0;
  for (int i = 0; i < 32; i++) m |= (unsigned)g_exchange[i] << i;
  __syncwarp();
  return m;
}
static int __popc(unsigned m) { return __builtin_popcount(m); }
static void __stcs(double *p, double x) { *p = x; }

#include "stores.h"
using namespace oco;

template <class F>
static void warp(F f) {
  pthread_barrier_init(&g_warp, nullptr, 32);
  std::vector<std::thread> lanes;
  for (unsigned l = 0; l < 32; l++)
    lanes.emplace_back([&, l] {
      threadIdx.x = l;
      f((int)l);
    });
  for (auto &t : lanes) t.join();
  pthread_barrier_destroy(&g_warp);
}

// Lanes that reach the reverse sweep while another still reads the forward sweep's shared memory.
extern "C" int stores_host_early_lanes() {
  RingSmem<double> ring;
  std::atomic<int> reading{32}, early{0};
  warp([&](int lane) {
    RingStores<true, double> st(OutPtrs{}, true, &ring);
    if (lane == 31) usleep(50000); // still in the forward sweep
    reading--;
    st.open(9);
    if (reading.load() != 0) early++; // from here on the lane may write the ring
  });
  return early.load();
}

// One warp's item of nz >= 4 levels in the order of the sweeps: rows of U (nz + 6), kappa and V (nz),
// urow and krow elements apart; level m of lane l is l * 1000 + m (V negative, kappa + 0.5).
template <bool ROWS>
static void item(int nz, int rows, double *U, double *K, double *V, int64_t urow, int64_t krow) {
  RingSmem<double> ring;
  warp([&](int lane) {
    const bool active = lane < rows;
    const int r = active ? lane : rows - 1;
    RingStores<ROWS, double> st(OutPtrs{U + r * urow, K + r * krow, V + r * krow, 1, 1, 1, urow, krow}, active, &ring);
    st.open(nz);
    auto u = [&](int m) { return lane * 1000.0 + m; };
    for (int q = 0; q < 6; q++) st.push_u(q, nz + 5 - q, u(nz + 5 - q));
    auto level = [&](int q, int m) { st.push(q, m, u(m), -u(m), u(m) + 0.5); };
    level(6, nz - 1);
    st.template group<false>(nz - 1, 7);
    int k = nz - 5;
    for (; k >= 7; k -= 8) {
      for (int q = 0; q < 8; q++) level(q, 3 + k - q);
      st.template group<true>(3 + k - 7, 8);
    }
    int q = 0;
    for (; k >= -3; k--) {
      level(q, 3 + k);
      if (++q == 8) {
        st.template group<false>(3 + k, 8);
        q = 0;
      }
    }
    st.finish(q);
  });
}
extern "C" void stores_host_item(int by_rows, int nz, int rows, double *U, double *K, double *V, int64_t urow, int64_t krow) {
  by_rows ? item<true>(nz, rows, U, K, V, urow, krow) : item<false>(nz, rows, U, K, V, urow, krow);
}
