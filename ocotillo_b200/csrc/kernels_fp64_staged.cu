/* kernels_fp64_staged.cu -- the staged FP64 solves of blocks and of ragged batches (see kernels_fp64.cu). */
#include "fp64_block.h"

namespace oco {

/* Batch records: thread i is record i of the dense [sum nz] list; its column comes from a
 * binary search of the nz prefix sums rec_pre[0..ncol]. */
__global__ void __launch_bounds__(PIL_THREADS) k_pillars_batch(const double *__restrict__ rho,
                                                               const double *__restrict__ T,
                                                               const MBatchCol *__restrict__ cols,
                                                               const int64_t *__restrict__ rec_pre, int64_t ncol,
                                                               int64_t n, double fully_ionized_T,
                                                               double *__restrict__ pil) {
  __shared__ double s_buf[PIL_THREADS / 32][32 * PIL_STRIDE];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t i0 = i - (threadIdx.x & 31);
  if (i0 >= n) return; /* whole warp past the end */
  double r[NF];
  if (i < n) {
    int64_t lo = 0, hi = ncol;
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (rec_pre[mid] <= i)
        lo = mid;
      else
        hi = mid;
    }
    const int64_t src = cols[lo].in_off + (i - rec_pre[lo]);
    pillar_record(rho[src], T[src], fully_ionized_T, 0, i != rec_pre[lo] && same_bits(T[src], T[src - 1]), r);
  } else {
#pragma unroll
    for (int k = 0; k < NF; k++) r[k] = 0.0; /* not stored */
  }
  store_pillars(r, s_buf[threadIdx.x >> 5], pil, i0, n);
}

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

/* ---- ragged batches (FP64 forms) -------------------------------------------------------- */
/* Item of a batch: wavelength w of column *c.  The descriptor is read through the read-only cache except,
 * in the ring kernels, its two counts, which the sweeps use throughout: as such loads they are repeated
 * there, and those kernels spill 112-168 bytes for it, 28-116 as plain ones (400 ragged columns, z fastest:
 * plain 2.94 -> 2.54 ms, stable 3.09 -> 2.98 ms; the lane-by-lane kernels lose 2-4% by plain loads). */
template <bool PLAIN>
struct BatchItem {
  const FP64BatchArgs &b;
  const MBatchCol *c;
  int64_t col;
  int w;
  __device__ __forceinline__ int nz() const { return PLAIN ? c->nz : __ldg(&c->nz); }
  __device__ __forceinline__ int nw() const { return PLAIN ? c->nw : __ldg(&c->nw); }
  __device__ __forceinline__ int iw() const { return w; }
  __device__ __forceinline__ const double *lam() const { return b.lam + __ldg(&c->lam_off); }
  __device__ __forceinline__ double dz() const { return __ldg(&c->dz); }
  __device__ __forceinline__ double dz2() const { return __ldg(&c->dz2); }
  __device__ __forceinline__ double dz1() const { return __ldg(&c->dz1); }
  __device__ __forceinline__ double sigma_grey() const { return 0.0; }
  __device__ __forceinline__ int64_t zoff(int64_t base, int rows) const { /* element z = 0 */
    return b.layout == 0 ? base + (int64_t)w * rows : base + w;
  }
  __device__ __forceinline__ double *U() const { return b.U ? b.U + zoff(__ldg(&c->u_off), nz() + 6) : nullptr; }
  __device__ __forceinline__ double *K() const { return b.K ? b.K + zoff(__ldg(&c->kv_off), nz()) : nullptr; }
  __device__ __forceinline__ double *V() const { return b.V ? b.V + zoff(__ldg(&c->kv_off), nz()) : nullptr; }
  __device__ __forceinline__ int64_t uz() const { return b.layout == 0 ? 1 : nw(); }
  __device__ __forceinline__ int64_t kz() const { return uz(); }
  __device__ __forceinline__ int64_t vz() const { return uz(); }
  __device__ __forceinline__ double *vtop() const { return b.Vtop ? b.Vtop + __ldg(&c->flux_off) + w : nullptr; }
  __device__ __forceinline__ double *vbot() const { return b.Vbot ? b.Vbot + __ldg(&c->flux_off) + w : nullptr; }
  __device__ __forceinline__ int64_t urow() const { return nz() + 6; }
  __device__ __forceinline__ int64_t krow() const { return nz(); }
  __device__ __forceinline__ int64_t ss() const { return 32; }
  __device__ __forceinline__ unsigned long long *status() const { return b.status; }
  __device__ __forceinline__ unsigned long long id() const { return ((unsigned long long)col << 32) | (unsigned)w; }
};

/* Warp-column tiling: tasks (column, 32-wavelength tile) from the device queue, longest
 * columns first; the column's records stream through the warp's shared-memory buffers and
 * the tile's wavelength constants sit in the warp's shared-memory table (as k_solve_staged). */
template <int FORM, int MODE>
__global__ void __launch_bounds__(128, 4) k_batch_fp64_staged(const FP64BatchArgs b) {
  __shared__ __align__(128) unsigned char s_warp[WARPS_PER_BLOCK * sizeof(StagedSmem)];
  StagedSmem &sm = reinterpret_cast<StagedSmem *>(s_warp)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t wbase = slot * 32 * (int64_t)b.max_nz + lane; /* each warp's scratch [z][lane], contiguous */
  double *gam = b.gam + wbase;
  double *uu = b.uu + wbase;
  double *kap = b.kap + wbase;
  double *qs = b.q + wbase;
  StagedPillars pa;
  init_staged(pa, sm);
  for (;;) {
    unsigned long long task = 0;
    if (lane == 0) task = atomicAdd(b.work, 1ull);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= (unsigned long long)b.ntasks) break;
    const uint2 t = b.tasks[task];
    const MBatchCol *c = b.cols + t.x;
    const int nw = __ldg(&c->nw);
    const int iw_raw = (int)t.y * 32 + lane;
    const bool active = iw_raw < nw;
    const int iw = active ? iw_raw : nw - 1;
    pa.nz = __ldg(&c->nz);
    pa.begin(b.pil + __ldg(&c->rec_off) * NF, lane);
    store_lam_shared(sm.lam, lane, b.lam + __ldg(&c->lam_off), iw, nw);
    __syncwarp();
    using Item = BatchItem<MODE == ST_RING>;
    const Item it{b, c, (int64_t)t.x, iw};
    solve_item<FORM, false, Item, StagedPillars, LamS>(it, active, pa, gam, uu, kap, qs, sm.lam,
                                                           TCacheS{sm.tc + lane},
                                                           make_stores<MODE, true, false>(out_ptrs(it), active, &sm.ring));
    if (__any_sync(0xffffffffu, pa.failed)) {
      if (lane == 0) atomicOr(&b.status[2], 1ull);
      pa.wait(0);
      pa.wait(1);
      return;
    }
  }
}

cudaError_t launch_pillars_batch(const double *rho, const double *T, const MBatchCol *cols, const int64_t *rec_pre,
                                 int64_t ncol, int64_t nrec, double fully_ionized_T, double *pil, cudaStream_t s) {
  if (nrec == 0) return cudaSuccess;
  k_pillars_batch<<<(unsigned)((nrec + PIL_THREADS - 1) / PIL_THREADS), PIL_THREADS, 0, s>>>(
      rho, T, cols, rec_pre, ncol, nrec, fully_ionized_T, pil);
  return cudaGetLastError();
}

template <int FORM>
static const void *block_fn(StoreMode m) {
  switch (m) {
    case ST_RING: return (const void *)k_solve_staged<FORM, ST_RING>;
    case ST_PLANES: return (const void *)k_solve_staged<FORM, ST_PLANES>;
    default: return (const void *)k_solve_staged<FORM, ST_LANE>;
  }
}
template <int FORM>
static const void *batch_fn(StoreMode m) {
  switch (m) {
    case ST_RING: return (const void *)k_batch_fp64_staged<FORM, ST_RING>;
    case ST_PLANES: return (const void *)k_batch_fp64_staged<FORM, ST_PLANES>;
    default: return (const void *)k_batch_fp64_staged<FORM, ST_LANE>;
  }
}
/* The order in which the kernels are named here is the order in which they are compiled, and the first three
 * of a unit come out differently (one register more or less, blocks laid out otherwise) and 2-9% slower:
 * a warm disk of 2744 columns x 448 levels x 68 wavelengths, stable, 5.19 and 5.65 ms.  So blocks and batches
 * share the unit, and the stable batch kernels, which lose least, come first. */
static const void *batch_stable_fn(StoreMode m) { return batch_fn<1>(m); }
const void *solve_staged_fn(int form, StoreMode m) { return form == 0 ? block_fn<0>(m) : block_fn<1>(m); }
static const void *batch_any_fn(int form, StoreMode m) { return form == 0 ? batch_fn<0>(m) : batch_stable_fn(m); }

cudaError_t launch_batch_fp64(const FP64BatchArgs &a, int form, int blocks, int threads, cudaStream_t s) {
  void *args[] = {(void *)&a};
  return cudaLaunchKernel(batch_any_fn(form, store_mode(a.U, a.K, a.V, a.layout)), dim3(blocks), dim3(threads), args, 0, s);
}

int batch_fp64_max_blocks_per_sm(int form, int threads) {
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_any_fn(form, ST_LANE), threads, 0);
  return (e == cudaSuccess && n > 0) ? n : 1;
}

}  // namespace oco
