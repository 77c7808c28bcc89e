/* kernels_fp64_items.cu -- the by-item FP64 block solve (see kernels_fp64.cu). */
#include "fp64_block.h"

namespace oco {

/* Generic path: warp tasks are 32 consecutive items of the flattened (column, lambda) index (lanes
 * past the last item repeat it and store nothing).  Bound by latency, so by the warps in flight: at
 * 202-208 registers two blocks fit an SM, three at 168 with some 50 bytes spilled (128 x 128 turbulent
 * columns x 256 levels, 17 wavelengths: plain, z fastest 4.35 -> 3.23 ms; stable 4.06 -> 3.07 ms with
 * lambda fastest, 4.48 -> 3.34 ms with z fastest).  FEW: two blocks hold every warp's task (solve_items_few),
 * so without the spills (23 x 61 columns x 991 levels x 17, stable 1.99 -> 1.92 ms). */
template <int FORM, bool GREY, int MODE, bool FEW>
__global__ void __launch_bounds__(128, FEW ? 1 : 3) k_solve(const SolveArgs a) {
  __shared__ RingSmem<double> s_ring[MODE == ST_RING ? WARPS_PER_BLOCK : 1];
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nitems = a.ncol * a.nw;
  const unsigned long long ntasks = (unsigned long long)((nitems + 31) / 32);
  const int64_t wbase = slot * 32 * (int64_t)a.nz + lane; /* each warp's scratch [z][lane], contiguous */
  double *gam = a.gam + wbase;
  double *uu = a.uu + wbase;
  double *kap = a.kap + wbase;
  double *qs = a.q + wbase;
  for (;;) {
    unsigned long long task = 0;
    if (lane == 0) task = atomicAdd(a.work, 1ull);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= ntasks) break;
    const bool active = (int64_t)task * 32 + lane < nitems;
    const int64_t item = active ? (int64_t)task * 32 + lane : nitems - 1;
    const int64_t cl = item / a.nw;
    const int iw = (int)(item - cl * a.nw);
    DirectPillars pa{a.pil + cl * (int64_t)a.nz * NF};
    const BlockItem it{a, cl, iw};
    solve_item<FORM, GREY, BlockItem, DirectPillars, LamR>(it, active, pa, gam, uu, kap, qs, nullptr, TCacheR{},
                                                           make_stores<MODE, false, false>(out_ptrs(it), active, &s_ring[MODE == ST_RING ? threadIdx.x >> 5 : 0]));
  }
}

/* planes: the lane-by-lane kernel stores no level either; grey, and plain lane by lane, take at most 168
 * registers, so one variant */
template <int FORM, bool GREY>
static const void *fn_of(StoreMode m, bool few) {
  if (m == ST_RING)
    return !GREY && few ? (const void *)k_solve<FORM, GREY, ST_RING, !GREY> : (const void *)k_solve<FORM, GREY, ST_RING, false>;
  constexpr bool F = !GREY && FORM == 1;
  return F && few ? (const void *)k_solve<FORM, GREY, ST_LANE, F> : (const void *)k_solve<FORM, GREY, ST_LANE, false>;
}
const void *solve_items_fn(int form, int grey, StoreMode m, bool few) {
  if (grey) return form == 0 ? fn_of<0, true>(m, few) : fn_of<1, true>(m, few);
  return form == 0 ? fn_of<0, false>(m, few) : fn_of<1, false>(m, few);
}

}  // namespace oco
