/* kernels_mixed_batch.cu -- the mixed solve of ragged batches (see kernels_mixed.cu). */
#include "mixed_block.h"

namespace oco {

/* ---- ragged batches ---------------------------------------------------------------------- */

/* Item of a batch: wavelength iw of column c. */
__device__ __forceinline__ MItem batch_item(const MixedBatchArgs &b, const MBatchCol &c, int iw) {
  MItem it;
  it.lam = b.lam + c.lam_off;
  it.nz = c.nz;
  it.nw = c.nw;
  it.iw = iw;
  it.dzf = c.dzf;
  it.ldz2i = c.ldz2i;
  it.ldz2f = c.ldz2f;
  it.dz2f = (float)c.dz2; /* as block_item's (float)(dz * dz) */
  it.dz1 = c.dz1;
  if (b.layout == 0) { /* per column [lambda][z] (z fastest) */
    it.o.U = b.U ? b.U + c.u_off + (int64_t)iw * (c.nz + 6) : nullptr;
    it.o.K = b.K ? b.K + c.kv_off + (int64_t)iw * c.nz : nullptr;
    it.o.V = b.V ? b.V + c.kv_off + (int64_t)iw * c.nz : nullptr;
    it.o.uz = it.o.kz = it.o.vz = 1;
  } else { /* per column [z][lambda] */
    it.o.U = b.U ? b.U + c.u_off + iw : nullptr;
    it.o.K = b.K ? b.K + c.kv_off + iw : nullptr;
    it.o.V = b.V ? b.V + c.kv_off + iw : nullptr;
    it.o.uz = it.o.kz = it.o.vz = c.nw;
  }
  it.o.urow = c.nz + 6;
  it.o.krow = c.nz;
  it.vtop = b.Vtop ? b.Vtop + c.flux_off + iw : nullptr;
  it.vbot = b.Vbot ? b.Vbot + c.flux_off + iw : nullptr;
  return it;
}

/* Warp-column tiling: tasks (column, 32-wavelength tile) from the device queue, longest
 * columns first; the column's records stream through the warp's shared-memory buffers. */
template <class SC, int MODE>
__global__ void __launch_bounds__(128, MBLOCKS) k_batch_mixed_staged(const MixedBatchArgs b) {
  __shared__ __align__(128) unsigned char s_warp[MWARPS * sizeof(MStagedSmem)];
  MStagedSmem &sm = reinterpret_cast<MStagedSmem *>(s_warp)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const SC sc{(char *)(b.s4 + slot * 32 * (int64_t)b.max_nz), lane}; /* the warp's scratch, contiguous */
  MStaged pa;
  init_staged(pa, sm);
  for (;;) {
    unsigned long long task = 0;
    if (lane == 0) task = atomicAdd(b.work, 1ull);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= (unsigned long long)b.ntasks) break;
    const uint2 t = b.tasks[task];
    const MBatchCol c = b.cols[t.x];
    const int iw_raw = (int)t.y * 32 + lane;
    const bool active = iw_raw < c.nw;
    const int iw = active ? iw_raw : c.nw - 1;
    pa.nz = c.nz;
    pa.begin(b.rec + c.rec_off * MZN);
    store_lam32_shared(sm.lam, lane, b.lam + c.lam_off, iw, c.nw);
    __syncwarp();
    const MItem it = batch_item(b, c, iw);
    const bool flag = msolve_item(it, active, pa, MLamS{sm.lam + lane}, sc, make_stores<MODE, true, false>(it.o, active, &sm.ring),
                                  b.repair_cond) ||
                      (active && __ldg(b.colflag + t.x) != 0u);
    if (__any_sync(0xffffffffu, pa.failed)) {
      if (lane == 0) atomicOr(&b.status[2], 1ull);
      pa.wait(0);
      pa.wait(1);
      return;
    }
    mark_tile(flag, (int64_t)t.x * b.rwstride + iw / 32, iw, ((unsigned long long)t.x << 32) | (unsigned)iw, b.rbits,
              b.rslot, b.rlist, b.rcount, b.ilist, b.icount);
  }
}

/* Packed tiling: the (column, wavelength) items of the columns sorted by nz (longest first)
 * form one list; a warp takes 32 consecutive items, so partial wavelength tiles of one column
 * are filled with the next column's items (similar nz, as the list is sorted). */
template <class SC>
__global__ void __launch_bounds__(128, 4) k_batch_mixed_packed(const MixedBatchArgs b) {
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const SC sc{(char *)(b.s4 + slot * 32 * (int64_t)b.max_nz), lane}; /* the warp's scratch, contiguous */
  for (;;) {
    unsigned long long task = 0;
    if (lane == 0) task = atomicAdd(b.work, 1ull);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= (unsigned long long)b.ntasks) break;
    const int64_t item = (int64_t)task * 32 + lane;
    bool flag = false;
    int32_t col = 0; /* a lane past the end solves column 0's first item without storing */
    int iw = 0;
    if (item < b.nitems) {
      int64_t lo = 0, hi = b.ncol; /* item_pre[lo] <= item < item_pre[hi] */
      while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (__ldg(b.item_pre + mid) <= item)
          lo = mid;
        else
          hi = mid;
      }
      col = __ldg(b.order + lo);
      iw = (int)(item - __ldg(b.item_pre + lo));
      const MBatchCol c = b.cols[col];
      MDirect pa{b.rec + c.rec_off * MZN};
      /* the lanes' columns differ in depth: each stores its own levels */
      const MItem it = batch_item(b, c, iw);
      flag = msolve_item(it, true, pa, load_lam32(it.lam, iw, it.nw), sc, LaneStores<false>(it.o, true), b.repair_cond) ||
             __ldg(b.colflag + col) != 0u;
    }
    mark_items(flag, (int64_t)col * b.rwstride + iw / 32, iw, ((unsigned long long)(unsigned)col << 32) | (unsigned)iw,
               b.rbits, b.rslot, b.rlist, b.rcount, b.ilist, b.icount);
  }
}

static const void *batch_mixed_fn(int tiling, StoreMode m) {
  if (tiling == BATCH_TILING_PACKED) return (const void *)k_batch_mixed_packed<MScratch12>;
  switch (m) {
    case ST_RING: return (const void *)k_batch_mixed_staged<MScratch12, ST_RING>;
    case ST_PLANES: return (const void *)k_batch_mixed_staged<MScratch12P, ST_PLANES>;
    default: return (const void *)k_batch_mixed_staged<MScratch12, ST_LANE>;
  }
}

int batch_mixed_max_blocks_per_sm(int tiling, int threads) {
  int n = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_mixed_fn(tiling, ST_LANE), threads, 0);
  if (e != cudaSuccess || n < 1) n = 1;
  return n;
}

cudaError_t launch_batch_mixed(const MixedBatchArgs &a, int tiling, int blocks, int threads, cudaStream_t s) {
  void *args[] = {(void *)&a};
  const StoreMode m = mixed_store_mode(a.U, a.K, a.V, a.layout, a.npoints, 1);
  return cudaLaunchKernel(batch_mixed_fn(tiling, m), dim3(blocks), dim3(threads), args, 0, s);
}

}  // namespace oco
