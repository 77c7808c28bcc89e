/*
 * kernels_fp64.cu -- the FP64 hot path on sm_100a.  Its kernels stand in one unit per path (records and
 * dispatch here; kernels_fp64_staged.cu, _items.cu, _split.cu), because a process loads a
 * unit's module, line tables included, when it first launches one of its kernels: as one unit of 14 MB,
 * which the compiler driver also compresses, that took 13.5 ms of a process's first solve, 2.2-3.7 ms so.
 *
 *   k_pillars   one thread per (column, z): Saha ionization and every factor of the
 *               reference's per-(z, lambda) opacity that depends on z only
 *               (gas_state.f90:30-110, continuous_opacity.f90:143-163 and the z-only
 *               parts of :203-300).  Hoisting changes no bits: each hoisted expression is
 *               the reference's expression with its operand order.
 *   k_solve     persistent kernel, one thread per (column, wavelength), warps take tasks
 *               of 32 consecutive items (lambda fastest) from a device counter.  Per item:
 *               opacity, albedo and source function (continuous_opacity.f90:175-201,
 *               :377-409), tridiagonal coefficients (auxiliary.f90:111-201), the Thomas
 *               forward sweep (auxiliary.f90:14-41) streaming gamma, u and kappa to a
 *               per-warp-slot scratch, then the back-substitution (:43-45), ghost zones
 *               (:49-62) and 6th-order flux (:64-109) in one reverse sweep with a 7-point
 *               register window.  All outputs leave in the reverse sweep (stores.h).
 *
 * Output stores (U, kappa, V and the emergent flux) use the streaming cache hint (st.global.cs,
 * evict first): they are never read back, and L2 then keeps more of the forward sweep's scratch
 * for the reverse sweep.
 *
 * These translation units are compiled with -fmad=false (no FMA contraction) and IEEE
 * division/square root, and call the ocomath functions, so FORM_PLAIN reproduces the CPU
 * oracle (ocomath back-end) bit for bit.  FORM_STABLE replaces the pivot recursion
 * bet_j = b_j - a_j*gam_j by its difference form (no cancellation; same linear system).
 */
#include <cuda_runtime.h>

#include "fp64_block.h"

namespace oco {

__global__ void __launch_bounds__(PIL_THREADS) k_pillars(const double *__restrict__ rho,
                                                         const double *__restrict__ T, int64_t n, int nz,
                                                         double fully_ionized_T, int grey,
                                                         double *__restrict__ pil, const ChunkInit init) {
  __shared__ double s_buf[PIL_THREADS / 32][32 * PIL_STRIDE];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  chunk_init(init, i, (int64_t)gridDim.x * blockDim.x);
  const int64_t i0 = i - (threadIdx.x & 31);
  if (i0 >= n) return; /* whole warp past the end */
  double r[NF];
#pragma unroll
  for (int k = 0; k < NF; k++) r[k] = 0.0; /* grey records set three fields */
  if (i < n) pillar_record(rho[i], T[i], fully_ionized_T, grey, i % nz != 0 && same_bits(T[i], T[i - 1]), r);
  store_pillars(r, s_buf[threadIdx.x >> 5], pil, i0, n);
}

cudaError_t launch_pillars(const double *rho, const double *T, int64_t ncol, int nz,
                           double fully_ionized_T, int grey, double *pil, const ChunkInit &init, cudaStream_t s) {
  int64_t n = ncol * nz;
  if (n == 0) return cudaSuccess;
  const int64_t blocks = (n + PIL_THREADS - 1) / PIL_THREADS;
  k_pillars<<<(unsigned)blocks, PIL_THREADS, 0, s>>>(rho, T, n, nz, fully_ionized_T, grey, pil, init);
  return cudaGetLastError();
}

bool solve_uses_staging(int nw) { return nw >= 64 || (nw % 32) == 0; }

static const void *solve_fn(int form, int grey, int nw, StoreMode m, bool few) {
  return !grey && solve_uses_staging(nw) ? solve_staged_fn(form, m) : solve_items_fn(form, grey, m, few);
}

int solve_fp64_max_blocks_per_sm(int form, int grey, int threads, int nw, StoreMode m, bool few) {
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, solve_fn(form, grey, nw, m, few), threads, 0);
  return (e == cudaSuccess && n > 0) ? n : 1;
}

/* Diagnostic: the staged kernels' bounded mbarrier wait, on a barrier phase that no copy or
 * arrival completes, so the wait runs out after `limit` polls and the timeout is reported in
 * status[2] as the solve kernels report it.  Nothing is in flight when the block exits. */
__global__ void k_bounded_wait_check(long long limit, unsigned long long *status) {
  __shared__ __align__(8) unsigned long long bar;
  const uint32_t b = smem_addr(&bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  long long spins = 0;
  bool done = true;
  while (!mbar_try_wait(b, 0u))
    if (++spins > limit) {
      done = false;
      break;
    }
  if (__any_sync(0xffffffffu, !done) && threadIdx.x == 0) atomicOr(&status[2], 1ull);
}

cudaError_t launch_bounded_wait_check(long long limit, unsigned long long *status, cudaStream_t s) {
  k_bounded_wait_check<<<1, 32, 0, s>>>(limit, status);
  return cudaGetLastError();
}

cudaError_t launch_solve_fp64(const SolveArgs &a, int form, int grey, int blocks, int threads, bool few, cudaStream_t s) {
  void *args[] = {(void *)&a};
  return cudaLaunchKernel(solve_fn(form, grey, a.nw, store_mode(a.U, a.K, a.V, a.layout), few), dim3(blocks),
                          dim3(threads), args, 0, s);
}

}  // namespace oco
