/* kernels_fp64_staged.cu -- the staged FP64 block solve (see kernels_fp64.cu). */
#include "fp64_block.h"

namespace oco {

/* Staged path: warp tasks are (column, tile of 32 wavelengths); the column's pillar records
 * are streamed into shared memory by bulk copies (see StagedPillars).  ST_RING: outputs with z fastest
 * through the ring (a warm disk of 1800 columns x 500 x 250, plain: 13.65 ms with lambda-fastest
 * temporaries and three transposes, 12.8 ms so; the AGN profile 4.8 ms, runs off the 64-byte
 * boundaries 6.4 ms; ragged batch of 400 columns with each lane storing its own rows 3.55 ms, 2.65
 * ms so).  With lambda fastest the warm disk takes 11.4 ms: the ring's instructions and the larger
 * code (instruction-cache misses) are the rest. */
template <int FORM, int MODE>
__global__ void __launch_bounds__(128, 4) k_solve_staged(const SolveArgs a) {
  __shared__ __align__(128) unsigned char s_warp[WARPS_PER_BLOCK * sizeof(StagedSmem)];
  StagedSmem &sm = reinterpret_cast<StagedSmem *>(s_warp)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int ntiles = (a.nw + 31) / 32;
  const unsigned long long ntasks = (unsigned long long)a.ncol * ntiles;
  const int64_t wbase = slot * 32 * (int64_t)a.nz + lane; /* each warp's scratch [z][lane], contiguous */
  double *gam = a.gam + wbase;
  double *uu = a.uu + wbase;
  double *kap = a.kap + wbase;
  double *qs = a.q + wbase;
  StagedPillars pa;
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
    pa.begin(a.pil + cl * (int64_t)a.nz * NF, lane);
    store_lam_shared(sm.lam, lane, a.lam, iw, a.nw);
    __syncwarp();
    const BlockItem it{a, cl, iw};
    solve_item<FORM, false, BlockItem, StagedPillars, LamS>(it, active, pa, gam, uu, kap, qs, sm.lam,
                                                          TCacheS{sm.tc + lane},
                                                          make_stores<MODE, true, false>(out_ptrs(it), active, &sm.ring));
    if (__any_sync(0xffffffffu, pa.failed)) {
      if (lane == 0) atomicOr(&a.status[2], 1ull);
      /* let copies still in flight land (bounded) before the block's shared memory is released */
      pa.wait(0);
      pa.wait(1);
      return;
    }
  }
}

template <int FORM>
static const void *fn_of(StoreMode m) {
  switch (m) {
    case ST_RING: return (const void *)k_solve_staged<FORM, ST_RING>;
    case ST_PLANES: return (const void *)k_solve_staged<FORM, ST_PLANES>;
    default: return (const void *)k_solve_staged<FORM, ST_LANE>;
  }
}
/* The stable form named first: the compiler then gives the plain kernel of LaneStores 126 registers
 * instead of 128 (297 tiles x 512 levels 0.41 instead of 0.43 ms). */
const void *solve_staged_fn(int form, StoreMode m) { return form == 1 ? fn_of<1>(m) : fn_of<0>(m); }

}  // namespace oco
