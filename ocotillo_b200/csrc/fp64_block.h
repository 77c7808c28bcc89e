/*
 * fp64_block.h -- what the FP64 solve kernels share besides the solve itself (fp64_core.h): the records'
 * stores, access to them (directly, or streamed into shared memory) and the (column, wavelength) item
 * of a block.
 */
#ifndef OCO_FP64_BLOCK_H
#define OCO_FP64_BLOCK_H

#include <cuda_runtime.h>

#include "fp64_core.h"

namespace oco {

#if defined(__CUDACC__) && !defined(__CUDACC_RTC__)
#if defined(__FMA__) || defined(__USE_FAST_MATH__)
#error "the FP64 kernels must be compiled without fast math"
#endif
#endif

constexpr int PIL_THREADS = 128;
constexpr int PIL_STRIDE = NF + 1; /* doubles per record in shared memory (odd: no bank conflicts) */

/* Writes the warp's records (lane l: record i0 + l, held in r) to pil with coalesced stores:
 * each lane puts its record in the warp's shared buffer, then the warp copies the 32
 * consecutive records out (records at or beyond n are not written). */
__device__ __forceinline__ void store_pillars(const double *r, double *__restrict__ buf, double *__restrict__ pil,
                                              int64_t i0, int64_t n) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NF; k++) buf[lane * PIL_STRIDE + k] = r[k];
  __syncwarp();
  double *o = pil + i0 * NF;
#pragma unroll
  for (int m = 0; m < NF; m++) {
    const int j = lane + 32 * m, q = j / NF, f = j % NF;
    if (i0 + q < n) o[j] = buf[q * PIL_STRIDE + f];
  }
}

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

/* ---- pillar access ------------------------------------------------------------------- */
/* Generic path: each lane reads its own column's records through the read-only cache. */
struct DirectPillars {
  const double *base;
  __device__ __forceinline__ GlobalRec at(int z) { return GlobalRec{base + (int64_t)z * NF}; }
};

constexpr int ZC = 12;            /* z records per staged chunk (static shared memory up to 48 KB) */
constexpr int WARPS_PER_BLOCK = 4; /* k_solve runs 128-thread blocks */
constexpr long long kSpinLimit = 1ll << 26;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

/* Staged path: all 32 lanes of the warp work on one column.  Lane 0 streams the column's
 * pillar records in chunks of ZC z with a bulk (TMA) copy into one of two shared-memory
 * buffers per warp; an mbarrier per buffer signals arrival.  Records are read in increasing
 * z, one at a time: entering chunk c frees the buffer of chunk c-1, which then receives
 * chunk c+1.  Waits are bounded; on timeout the warp records the failure and stops. */
struct StagedPillars {
  PillarRecord *buf; /* shared: [2][ZC] */
  uint32_t bar0;  /* shared address of two mbarriers (8 B each) */
  const double *src;
  const PillarRecord *rec; /* next record, left of them in the buffer */
  int nz, nchunks, cur, left;
  uint32_t waits;    /* bit b: parity of the next wait on buffer b */
  uint32_t inflight; /* bit b: a copy into buffer b has been issued and not yet waited for */
  bool failed;

  __device__ __forceinline__ void issue(int c) {
    const int rows = min(ZC, nz - c * ZC);
    const uint32_t bytes = (uint32_t)(rows * NF * sizeof(double));
    const uint32_t bar = bar0 + 8u * (c & 1);
    const uint32_t dst = smem_addr(buf + (c & 1) * ZC);
    const size_t g = __cvta_generic_to_global(src + (int64_t)c * ZC * NF);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(g), "r"(bytes), "r"(bar)
                 : "memory");
  }
  /* Waits (bounded) for the copy into buffer b.  Every lane tracks the same state. */
  __device__ __forceinline__ bool wait(int b) {
    if (!((inflight >> b) & 1u)) return true;
    const uint32_t bar = bar0 + 8u * b;
    const uint32_t parity = (waits >> b) & 1u;
    long long spins = 0;
    while (!mbar_try_wait(bar, parity))
      if (++spins > kSpinLimit) return false;
    waits ^= 1u << b;
    inflight &= ~(1u << b);
    return true;
  }
  __device__ __forceinline__ void note_issue(int c) { inflight |= 1u << (c & 1); }
  __device__ __forceinline__ void begin(const double *column, int lane) {
    src = column;
    cur = -1;
    left = 0;
    nchunks = (nz + ZC - 1) / ZC;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); /* this lane's tile accesses before the copies */
    __syncwarp();
    if (lane == 0) issue(0);
    note_issue(0);
  }
  /* The next record; z counts up from 0. */
  __device__ __forceinline__ SharedRec at(int) {
    if (left == 0) {
      const int c = ++cur;
      __syncwarp();
      if (!failed && c + 1 < nchunks) {
        if ((threadIdx.x & 31) == 0) issue(c + 1);
        note_issue(c + 1);
      }
      if (!failed && !wait(c & 1)) failed = true;
      rec = buf + (c & 1) * ZC;
      left = ZC;
    }
    left--;
    const SharedRec r{rec};
    rec++;
    return r;
  }
};

/* What one (column, wavelength) item needs besides its records, as an accessor read on
 * demand (kernel parameters and descriptors stay in their state spaces instead of registers).
 * Block kernels: column cl of the chunk, wavelength iw. */
struct BlockItem {
  const SolveArgs &a;
  int64_t cl;
  int w;
  __device__ __forceinline__ int64_t idx() const {
    return (a.layout == 0) ? (int64_t)w * a.ld_col + a.c_off + cl : (a.c_off + cl) * a.nw + w;
  }
  __device__ __forceinline__ int64_t pidx() const { return (int64_t)w * a.ld_col + a.c_off + cl; }
  __device__ __forceinline__ const double *lam() const { return a.lam; }
  __device__ __forceinline__ int nz() const { return a.nz; }
  __device__ __forceinline__ int nw() const { return a.nw; }
  __device__ __forceinline__ int iw() const { return w; }
  __device__ __forceinline__ double dz() const { return a.dz; }
  __device__ __forceinline__ double dz2() const { return a.dz2; }
  __device__ __forceinline__ double dz1() const { return a.dz1; }
  __device__ __forceinline__ double sigma_grey() const { return a.sigma_grey; }
  __device__ __forceinline__ double *U() const { return a.U ? a.U + idx() * a.U_is : nullptr; }
  __device__ __forceinline__ double *K() const { return a.K ? a.K + idx() * a.K_is : nullptr; }
  __device__ __forceinline__ double *V() const { return a.V ? a.V + idx() * a.V_is : nullptr; }
  __device__ __forceinline__ int64_t uz() const { return a.U_zs; }
  __device__ __forceinline__ int64_t kz() const { return a.K_zs; }
  __device__ __forceinline__ int64_t vz() const { return a.V_zs; }
  __device__ __forceinline__ double *vtop() const { return a.Vtop ? a.Vtop + pidx() : nullptr; }
  __device__ __forceinline__ double *vbot() const { return a.Vbot ? a.Vbot + pidx() : nullptr; }
  /* z fastest: elements between the rows of neighbouring wavelengths */
  __device__ __forceinline__ int64_t urow() const { return a.ld_col * a.U_is; }
  __device__ __forceinline__ int64_t krow() const { return a.ld_col * (int64_t)a.nz; }
  __device__ __forceinline__ int64_t ss() const { return 32; }
  __device__ __forceinline__ unsigned long long *status() const { return a.status; }
  __device__ __forceinline__ unsigned long long id() const {
    return (unsigned long long)((a.c_off + cl) * a.nw + w);
  }
};

template <class IT>
__device__ __forceinline__ OutPtrs out_ptrs(const IT &it) {
  return OutPtrs{it.U(), it.K(), it.V(), it.uz(), it.kz(), it.vz(), it.urow(), it.krow()};
}

/* A staged warp's shared memory.  The reverse sweep needs none of the forward sweep's: its output
 * ring takes it over (the next task rewrites it, the buffers by bulk copies ordered after the
 * ring's last use by the fence in StagedPillars::begin). */
struct StagedSmem {
  union {
    struct {
      PillarRecord pil[2 * ZC];
      double lam[NLF * 32];     /* the task's 32 wavelengths' constants */
      double2 tc[NTC / 2 * 32]; /* the lanes' temperature factors */
    };
    RingSmem<double> ring;
  };
  unsigned long long bar[2];
  __device__ StagedSmem() = delete;
};
static_assert(sizeof(StagedSmem) % 16 == 0, "bulk copies and 16-byte pairs");

__device__ __forceinline__ void init_staged(StagedPillars &pa, StagedSmem &sm) {
  pa.buf = sm.pil;
  pa.bar0 = smem_addr(&sm.bar[0]);
  pa.waits = 0;
  pa.inflight = 0;
  pa.failed = false;
  if ((threadIdx.x & 31) == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(pa.bar0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(pa.bar0 + 8u) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
}

}  // namespace oco

#endif /* OCO_FP64_BLOCK_H */
