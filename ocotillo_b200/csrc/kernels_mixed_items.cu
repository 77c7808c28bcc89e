/* kernels_mixed_items.cu -- the by-item mixed block solve (see kernels_mixed.cu). */
#include "mixed_block.h"

namespace oco {

/* Few wavelengths: 32 consecutive items per warp (lanes past the last item repeat it and store
 * nothing).  FEW: every warp has its task at four blocks per SM (mixed_items_few), at 126 registers and with
 * kappa leaving in the reverse sweep; otherwise five blocks at 96 registers with 28 bytes spilled and kappa
 * leaving in the forward sweep.  Few / other, lambda fastest, us: 16 columns x 500 levels x 17 wavelengths
 * 380 / 430 (AGN), 567 / 617 (turbulent); 128 x 128 x 256 turbulent, 5 wavelengths 1336 / 1056, 17 2070 /
 * 1890, 33 3234 / 2970.  The ring variant spills twice as much at five blocks and gains at 5 wavelengths
 * only (1.41 -> 1.23 ms; 3 1.04 -> 1.15 ms, 17 and 33 the same): four. */
template <class SC, int MODE, bool FEW>
__global__ void __launch_bounds__(128, MODE == ST_RING || FEW ? 4 : 5) k_solve_mixed(const MixedArgs a) {
  __shared__ RingSmem<float> s_ring[MODE == ST_RING ? MWARPS : 1];
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nitems = a.ncol * a.nw;
  const unsigned long long ntasks = (unsigned long long)((nitems + 31) / 32);
  const SC sc{(char *)(a.s4 + slot * 32 * (int64_t)a.nz), lane}; /* the warp's scratch, contiguous */
  for (;;) {
    unsigned long long task = 0;
    if (lane == 0) task = atomicAdd(a.work, 1ull);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= ntasks) break;
    const bool active = (int64_t)task * 32 + lane < nitems;
    const int64_t item = active ? (int64_t)task * 32 + lane : nitems - 1;
    const int64_t cl = item / a.nw;
    const int iw = (int)(item - cl * a.nw);
    MDirect pa{a.rec + cl * (int64_t)a.nz * MZN};
    const MItem it = block_item(a, cl, iw);
    const bool flag = msolve_item(it, active, pa, load_lam32(it.lam, iw, it.nw), sc,
                                  make_stores<MODE, false, FEW>(it.o, active, &s_ring[MODE == ST_RING ? threadIdx.x >> 5 : 0]), a.repair_cond) ||
                      (active && __ldg(a.colflag + cl) != 0u);
    mark_items(flag, cl * ((a.nw + 31) / 32) + iw / 32, iw, (unsigned long long)item, a.rbits, a.rslot, a.rlist, a.rcount,
               a.ilist, a.icount);
  }
}

const void *solve_mixed_items_fn(StoreMode m, bool few) {
  if (m == ST_RING) return (const void *)k_solve_mixed<MScratch16, ST_RING, false>;
  return few ? (const void *)k_solve_mixed<MScratch16, ST_LANE, true> : (const void *)k_solve_mixed<MScratch16, ST_LANE, false>;
}

}  // namespace oco
