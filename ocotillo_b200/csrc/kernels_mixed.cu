/*
 * kernels_mixed.cu -- the mixed-precision form (OCO_FORM_MIXED) on sm_100a.
 *
 *   k_solve_mixed     persistent kernel, one thread per (column, wavelength); warp tasks are
 *                     (column, 32 wavelengths) with the column's records streamed into shared
 *                     memory by bulk copies (TMA, mbarrier, bounded waits), or 32 consecutive
 *                     items with direct loads when nw is small.  Forward sweep: log2-space
 *                     opacity, scaled rows and the difference-form Thomas elimination in FP32
 *                     (the source function's exponent as integer + FP32 fraction),
 *                     writing a scratch record per z (|gamma| or q, kappa or 1/kappa, u mantissa
 *                     and exponent); reverse sweep: extended-range FP32 back-substitution, the
 *                     differences D_j, and the flux from a 6-value window of differences, with
 *                     FP64 outputs (stores.h).
 * See mixed_core.h for the arithmetic and its relation to the reference.
 */
#include <cuda_runtime.h>

#include "mixed_block.h"

namespace oco {

/* ST_RING: outputs with z fastest through the ring (AGN grid of 1600 columns x 512 x 256: 5.04 ms with
 * lambda-fastest temporaries and three transposes, 3.43 ms so; with lambda fastest 2.95 ms). */
template <class SC, int MODE>
__global__ void __launch_bounds__(128, MBLOCKS) k_solve_mixed_staged(const MixedArgs a) {
  __shared__ __align__(128) unsigned char s_warp[MWARPS * sizeof(MStagedSmem)];
  MStagedSmem &sm = reinterpret_cast<MStagedSmem *>(s_warp)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int ntiles = (a.nw + 31) / 32;
  const unsigned long long ntasks = (unsigned long long)a.ncol * ntiles;
  const SC sc{(char *)(a.s4 + slot * 32 * (int64_t)a.nz), lane}; /* the warp's scratch, contiguous */
  MStaged pa;
  pa.nz = a.nz;
  init_staged(pa, sm);
  for (;;) {
    unsigned long long task = 0;
    if (lane == 0) task = atomicAdd(a.work, 1ull);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= ntasks) break;
    const int64_t cl = (int64_t)(task / ntiles);
    const int tile = (int)(task - (unsigned long long)cl * ntiles);
    const int iw_raw = tile * 32 + lane;
    const bool active = iw_raw < a.nw;
    const int iw = active ? iw_raw : a.nw - 1;
    pa.begin(a.rec + cl * (int64_t)a.nz * MZN);
    store_lam32_shared(sm.lam, lane, a.lam, iw, a.nw);
    __syncwarp();
    const MItem it = block_item(a, cl, iw);
    const bool flag = msolve_item(it, active, pa, MLamS{sm.lam + lane}, sc, make_stores<MODE, true, false>(it.o, active, &sm.ring),
                                  a.repair_cond) ||
                      (active && __ldg(a.colflag + cl) != 0u);
    if (__any_sync(0xffffffffu, pa.failed)) {
      if (lane == 0) atomicOr(&a.status[2], 1ull);
      pa.wait(0);
      pa.wait(1);
      return;
    }
    mark_tile(flag, cl * ntiles + iw / 32, iw, (unsigned long long)(cl * a.nw + iw), a.rbits, a.rslot, a.rlist,
              a.rcount, a.ilist, a.icount);
  }
}

static bool mixed_uses_staging(int nw) { return (nw >= 64) || (nw % 32) == 0; }

static const void *solve_mixed_fn(int nw, StoreMode m, bool few) {
  if (mixed_uses_staging(nw)) switch (m) {
      case ST_RING: return (const void *)k_solve_mixed_staged<MScratch16, ST_RING>;
      case ST_PLANES: return (const void *)k_solve_mixed_staged<MScratch12P, ST_PLANES>;
      default: return (const void *)k_solve_mixed_staged<MScratch16, ST_LANE>;
    }
  return solve_mixed_items_fn(m, few);
}

int solve_mixed_max_blocks_per_sm(int threads, int nw, StoreMode m, bool few) {
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, solve_mixed_fn(nw, m, few), threads, 0);
  return (e == cudaSuccess && n > 0) ? n : 1;
}

cudaError_t launch_solve_mixed(const MixedArgs &a, int blocks, int threads, bool few, cudaStream_t s) {
  void *args[] = {(void *)&a};
  const StoreMode m = mixed_store_mode(a.U, a.K, a.V, a.layout, a.ncol * a.nw, a.nz);
  return cudaLaunchKernel(solve_mixed_fn(a.nw, m, few), dim3(blocks), dim3(threads), args, 0, s);
}

}  // namespace oco
