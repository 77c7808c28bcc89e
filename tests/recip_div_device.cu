// recip_div.h on the device for tests/test_gpu_recip_div.py: reciprocals and quotients against the division
// operator.  One thread per pattern of a divisor's 20 leading fraction bits (the seed's argument), with
// random bits below and random exponents; the dividends are random, or next to a midpoint between two
// quotients.
#include <cstdint>

#include <cuda_runtime.h>

#include "recip_div.h"

static __device__ uint64_t mix(uint64_t x) { // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

// count[0]: pairs used; [1]: wrong reciprocals; [2]: wrong quotients; [3]: seeds off by 2^-19 or more.
__global__ void k_check(uint64_t seed, unsigned long long *count) {
  const uint64_t hi = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; // < 2^20
  uint64_t used = 0, bad_r = 0, bad_q = 0, bad_s = 0;
  for (int rep = 0; rep < 16; rep++) {
    const uint64_t r0 = mix(seed + hi * 64 + rep * 4), r1 = mix(r0), r2 = mix(r1);
    const uint64_t low = rep == 0 ? 0 : rep == 1 ? 0xffffffffull : r0 & 0xffffffffull;
    const int eb = (int)(r1 % 400) - 200, ea = (int)((r1 >> 32) % 1238) - 759;
    const double m = __longlong_as_double((long long)((1023ull << 52) | (hi << 32) | low));
    const double b = ldexp((r2 & 1) ? -m : m, eb);
    double a = __longlong_as_double((long long)((1023ull << 52) | (r2 >> 12)));
    if (rep & 1) { // near m (q + half an ulp)
      const double t = fma(m, 0x1p-53, 0.0);
      a = fma(m, a, t);
      a = (r0 >> 40) & 1 ? a : __longlong_as_double(__double_as_longlong(a) + ((r0 >> 41) & 1 ? 1 : -1));
    }
    a = ldexp(a, ea);
    if (!div_b_ok(b) || !div_a_ok(a)) continue;
    used++;
    const double y = div_recip(b);
    bad_s += !(fabs(fma(-b, div_seed(b), 1.0)) < 0x1p-19);
    bad_r += __double_as_longlong(y) != __double_as_longlong(1.0 / b);
    bad_q += __double_as_longlong(div_quot(a, b, y)) != __double_as_longlong(a / b);
  }
  atomicAdd(&count[0], (unsigned long long)used);
  if (bad_r) atomicAdd(&count[1], (unsigned long long)bad_r);
  if (bad_q) atomicAdd(&count[2], (unsigned long long)bad_q);
  if (bad_s) atomicAdd(&count[3], (unsigned long long)bad_s);
}

extern "C" int recip_div_device(uint64_t seed, uint64_t *out) {
  unsigned long long *d = nullptr;
  cudaError_t e = cudaMalloc((void **)&d, 4 * sizeof *d);
  if (e == cudaSuccess) e = cudaMemset(d, 0, 4 * sizeof *d);
  if (e == cudaSuccess) {
    k_check<<<(1 << 20) / 256, 256>>>(seed, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d, 4 * sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
