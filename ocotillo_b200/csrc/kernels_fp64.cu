/*
 * kernels_fp64.cu -- the FP64 hot path on sm_100a.
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
 * This translation unit is compiled with -fmad=false (no FMA contraction) and IEEE
 * division/square root, and calls the ocomath functions, so FORM_PLAIN reproduces the CPU
 * oracle (ocomath back-end) bit for bit.  FORM_STABLE replaces the pivot recursion
 * bet_j = b_j - a_j*gam_j by its difference form (no cancellation; same linear system).
 */
#include <cuda_runtime.h>

#include "fp64_core.h"

namespace oco {

#if defined(__CUDACC__) && !defined(__CUDACC_RTC__)
#if defined(__FMA__) || defined(__USE_FAST_MATH__)
#error "kernels_fp64.cu must be compiled without fast math"
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

/* Generic path: warp tasks are 32 consecutive items of the flattened (column, lambda) index (lanes
 * past the last item repeat it and store nothing).  Bound by latency, so by the warps in flight: at
 * 202-208 registers two blocks fit an SM, three at 168 with some 50 bytes spilled (128 x 128 turbulent
 * columns x 256 levels, 17 wavelengths: plain, z fastest 4.35 -> 3.23 ms; stable 4.06 -> 3.07 ms with
 * lambda fastest, 4.48 -> 3.34 ms with z fastest). */
template <int FORM, bool GREY, int MODE>
__global__ void __launch_bounds__(128, 3) k_solve(const SolveArgs a) {
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

/* ---- the split block solve ------------------------------------------------------------- */
/* With few items the persistent kernels leave most of the GPU idle while each warp walks its column
 * alone (2 us per level and warp, whatever the number of warps: 16 columns x 500 x 250 took 1.03
 * ms, 0.45 ms after the sweep's own changes).  Here everything that is independent along z runs
 * first, parallel over (warp tile, RZ levels): k_rows writes the rows' coefficients; k_chain then
 * runs the recurrences, one warp per tile, with nothing but them on its serial chain: 0.23 ms for
 * those 16 columns.  That moves ~180 B per point instead of ~75, so it is taken while there are at
 * most two tiles per SM (solve_is_split; a full wave of the persistent kernel holds 16), and for
 * grey transfer always: it has one wavelength per column (few items) and no opacity sums, and reads
 * rho and T directly instead of a 208-byte record per cell (16,384 columns x 512: 1.08 -> 0.43 ms).
 * Per point the operations are solve_item's, so the same bits. */
constexpr int RZ = 8; /* levels per warp of k_rows: two more are computed for the neighbours */

/* One cell of a grey column (grey_parameters, continuous_opacity.f90:377-390); the factors of an
 * unchanged temperature are kept. */
struct GreyCell {
  double t, p35, S;
};
template <bool STABLE>
__device__ __forceinline__ Opac opacity_grey_cell(double r, double t, double sg, bool fresh, GreyCell &k) {
  if (fresh || !same_bits(t, k.t)) {
    const double t2 = t * t;
    k.t = t;
    k.S = sigma_sb * (t2 * t2);
    k.p35 = 3.68e22 * oco_pow(t, -3.5);
  }
  const double alpha = k.p35 * r, tot = alpha + sg;
  Opac o;
  o.op = tot * r;
  o.S = k.S;
  o.num = STABLE ? alpha : sg;
  o.kr = tot;
  const double q = div_quot(o.num, tot, div_recip(tot));
  o.w = STABLE ? q : 1.0 - q;
  o.wok = div_b_ok(tot) & div_a_ok(o.num);
  o.ook = op_ok(o.op);
  return o;
}

/* The item of a lane: TILE, wavelength tile*32 + lane of the tile's column, otherwise item
 * tile*32 + lane of the flattened list; lanes past the end repeat the last. */
template <bool TILE>
__device__ __forceinline__ bool split_item(const SolveArgs &a, int64_t t, int64_t &cl, int &iw) {
  const int lane = threadIdx.x & 31;
  if (TILE) {
    const int ntiles = (a.nw + 31) / 32;
    cl = t / ntiles;
    iw = (int)(t - cl * ntiles) * 32 + lane;
    const bool on = iw < a.nw;
    if (!on) iw = a.nw - 1;
    return on;
  }
  const int64_t n = a.ncol * a.nw, i = t * 32 + lane, item = i < n ? i : n - 1;
  cl = item / a.nw;
  iw = (int)(item - cl * a.nw);
  return i < n;
}

/* Coefficient arrays of the tiles: [tile][z][32], in this order after one another; at level z0 of
 * tile t. */
struct SplitRows {
  double *aa, *xx, *cc, *dd, *kap; /* xx: diagonal (plain), its excess (stable); kap as the sweep's scratch */
  __device__ __forceinline__ SplitRows(const SolveArgs &a, int64_t tiles, int64_t t, int z0) {
    const int64_t plane = tiles * 32 * a.nz;
    aa = a.gam + t * 32 * a.nz + tile_level(z0) + (threadIdx.x & 31);
    xx = aa + plane;
    cc = xx + plane;
    dd = cc + plane;
    kap = dd + plane;
  }
};

template <int FORM, bool GREY, bool REF, bool TILE>
__global__ void __launch_bounds__(128, 4) k_rows(const SolveArgs a, int64_t tiles, const ChunkInit init) {
  chunk_init(init, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
  const int nch = (a.nz + RZ - 1) / RZ;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= tiles * nch) return;
  const int64_t t = w / nch;
  const int nz = a.nz, z0 = (int)(w - t * nch) * RZ, z1 = min(z0 + RZ, nz);
  int64_t cl;
  int iw;
  const bool active = split_item<TILE>(a, t, cl, iw);
  const BlockItem it{a, cl, iw};
  const LamR L(it, nullptr, !GREY);
  TCacheR tc;
  GreyCell gc;
  const SplitRows S(a, tiles, t, z0);
  const int zf = max(z0 - 1, 0); /* first level computed */
  auto opac = [&](int z) -> Opac {
    Opac o;
    if constexpr (GREY)
      o = opacity_grey_cell<FORM == 1>(__ldg(a.rho + cl * nz + z), __ldg(a.T + cl * nz + z), a.sigma_grey, z == zf, gc);
    else
      o = opacity_at<FORM == 1>(GlobalRec{a.pil + (cl * (int64_t)nz + z) * NF}, L, tc, z == zf);
    settle_opac<FORM == 1>(o);
    return o;
  };
  const double dz = a.dz, dz2 = a.dz2;
  double *Kb = REF || !active ? nullptr : it.K();
  const int64_t kz = it.kz();
  double kh = 1.0, yk = 1.0; /* mean opacity below the level */
  int okk = 0;
  Opac cur = opac(zf);
  auto mean = [&](const Opac &lo, const Opac &hi) {
    kh = 0.5 * (hi.op + lo.op);
    yk = div_recip(kh);
    okk = lo.ook & hi.ook & div_b_frac_ok(kh);
  };
  if (z0 > 0) {
    const Opac up = opac(z0);
    mean(cur, up);
    cur = up;
  }
  for (int j = z0; j < z1; j++) {
    const int i = (j - z0) * 32;
    const double op = cur.op, o2 = op * op;
    double o1 = div_recip(op);
    if (!cur.ook) o1 = div_call(1.0, op);
    Opac nxt{};
    if (j == 0 || j == nz - 1) { /* fill_boundary_coeffs :187-197 */
      const double zt = ((op * dz2) * cur.w) * 0.25;
      S.dd[i] = -((cur.S * zt) * o2);
      S.xx[i] = FORM == 0 ? -(((o1 + dz) + zt) * o2) : (dz + zt) * o2;
      S.aa[i] = op; /* row 0: unused */
      S.cc[i] = j == 0 ? op : 0.0;
      if (j == 0) {
        nxt = opac(1);
        mean(cur, nxt);
      }
    } else { /* fill_center_coeffs :159-165 */
      nxt = opac(j + 1);
      double aa = div_quot(o2, kh, yk);
      if (!okk) aa = div_call(o2, kh);
      mean(cur, nxt);
      double cc = div_quot(o2, kh, yk);
      if (!okk) cc = div_call(o2, kh);
      const double z3 = (dz2 * (op * (op * op))) * cur.w;
      S.aa[i] = aa;
      S.cc[i] = cc;
      S.xx[i] = FORM == 0 ? -((aa + cc) + z3) : z3;
      S.dd[i] = -(cur.S * z3);
    }
    S.kap[i] = REF ? op : o1;
    if (Kb) __stcs(&Kb[j * kz], op);
    cur = nxt;
  }
}

/* One warp per block, so that the tiles spread over the SMs. */
template <int FORM, bool REF, bool TILE>
__global__ void __launch_bounds__(32) k_chain(const SolveArgs a, int64_t tiles) {
  __shared__ RingSmem<double> s_ring[1];
  const int64_t t = blockIdx.x;
  const int nz = a.nz;
  int64_t cl;
  int iw;
  const bool active = split_item<TILE>(a, t, cl, iw);
  const BlockItem it{a, cl, iw};
  const SplitRows S(a, tiles, t, 0);
  bool bad = false;
  Chain e = chain_first<FORM>(S.xx[0], S.cc[0], S.dd[0], bad);
  S.dd[0] = e.u;
  auto step = [&](int j, double aa, double xx, double cc, double dd) {
    double g, q;
    chain_step<FORM>(e, aa, xx, cc, dd, g, q, bad);
    S.aa[tile_level(j)] = g;
    S.dd[tile_level(j)] = e.u;
    if (FORM == 1) S.xx[tile_level(j - 1)] = q; /* q_{j-1} over the excess of row j - 1 */
  };
  constexpr int G = RG_ALONE;
  struct Row {
    double a, x, c, d;
  } A[G], B[G];
  auto load = [&](Row *l, int j0) {
#pragma unroll
    for (int i = 0; i < G; i++) {
      const int64_t k = tile_level(min(j0 + i, nz - 1));
      l[i] = Row{S.aa[k], S.xx[k], S.cc[k], S.dd[k]};
    }
  };
  auto steps = [&](const Row *l, int j0) {
#pragma unroll
    for (int i = 0; i < G; i++) step(j0 + i, l[i].a, l[i].x, l[i].c, l[i].d);
  };
  int j = 1;
  load(A, 1);
#pragma unroll 1
  for (; j + 2 * G <= nz && nz >= LONG_NZ; j += 2 * G) {
    load(B, j + G);
    steps(A, j);
    load(A, j + 2 * G);
    steps(B, j + G);
  }
  Row x = A[0];
#pragma unroll 1
  for (; j < nz; j++) { /* one level loaded ahead */
    const int64_t k = tile_level(min(j + 1, nz - 1));
    const Row nx{S.aa[k], S.xx[k], S.cc[k], S.dd[k]};
    step(j, x.a, x.x, x.c, x.d);
    x = nx;
  }
  if (active && bad) {
    atomicAdd(&it.status()[0], 1ull);
    atomicMin(&it.status()[1], it.id());
  }
  __syncwarp();
  auto st = make_stores<REF ? ST_RING : ST_LANE, TILE, false>(out_ptrs(it), active, s_ring);
  solve_reverse<FORM, RG_ALONE>(it, active, e.u, S.aa, S.dd, S.kap, S.xx, st);
}

static bool split_by_tile(int nw) { return nw >= 64 || nw % 32 == 0; }
int64_t split_tiles(int64_t ncol, int nw) {
  return split_by_tile(nw) ? ncol * ((nw + 31) / 32) : (ncol * nw + 31) / 32;
}
bool solve_is_split(int grey, int64_t ncol, int nw, int num_sms) {
  return grey || split_tiles(ncol, nw) <= 2 * (int64_t)num_sms;
}

/* Outputs with z fastest: through the ring only where they do not fit in L2, which otherwise joins the
 * lanes' own stores into whole lines for nothing (16 columns x 500 x 250, 48 MB: 0.33 ms with the
 * ring, 0.23 ms without; 16,384 grey columns, 201 MB: 0.44 and 0.42 ms). */
constexpr int64_t SPLIT_RING_BYTES = 256ll << 20;

template <int FORM, bool GREY, bool REF, bool TILE>
static cudaError_t split_launch(const SolveArgs &a, const ChunkInit &init, cudaStream_t s) {
  const int64_t tiles = split_tiles(a.ncol, a.nw), warps = tiles * ((a.nz + RZ - 1) / RZ);
  k_rows<FORM, GREY, REF, TILE><<<(unsigned)((warps + 3) / 4), 128, 0, s>>>(a, tiles, init);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_chain<FORM, REF, TILE><<<(unsigned)tiles, 32, 0, s>>>(a, tiles);
  return cudaGetLastError();
}
template <int FORM, bool REF>
static cudaError_t split_launch(const SolveArgs &a, int grey, const ChunkInit &init, cudaStream_t s) {
  if (grey) return split_launch<FORM, true, REF, false>(a, init, s);
  return split_by_tile(a.nw) ? split_launch<FORM, false, REF, true>(a, init, s)
                             : split_launch<FORM, false, REF, false>(a, init, s);
}
/* init: set up by k_rows where no record kernel comes before it (grey). */
cudaError_t launch_solve_split(const SolveArgs &a, int form, int grey, const ChunkInit &init, cudaStream_t s) {
  if (a.layout == 0 && split_tiles(a.ncol, a.nw) * 32 * (int64_t)a.nz * 24 > SPLIT_RING_BYTES)
    return form == 0 ? split_launch<0, true>(a, grey, init, s) : split_launch<1, true>(a, grey, init, s);
  return form == 0 ? split_launch<0, false>(a, grey, init, s) : split_launch<1, false>(a, grey, init, s);
}

/* ---- ragged batches (FP64 forms) -------------------------------------------------------- */
/* Item of a batch: wavelength w of column *c (descriptor read through the read-only cache). */
struct BatchItem {
  const FP64BatchArgs &b;
  const MBatchCol *c;
  int64_t col;
  int w;
  __device__ __forceinline__ int nz() const { return __ldg(&c->nz); }
  __device__ __forceinline__ int nw() const { return __ldg(&c->nw); }
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
    const BatchItem it{b, c, (int64_t)t.x, iw};
    solve_item<FORM, false, BatchItem, StagedPillars, LamS>(it, active, pa, gam, uu, kap, qs, sm.lam,
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
static const void *batch_fn_of(StoreMode m) {
  switch (m) {
    case ST_RING: return (const void *)k_batch_fp64_staged<FORM, ST_RING>;
    case ST_PLANES: return (const void *)k_batch_fp64_staged<FORM, ST_PLANES>;
    default: return (const void *)k_batch_fp64_staged<FORM, ST_LANE>;
  }
}
static const void *batch_fn(int form, StoreMode m) { return form == 0 ? batch_fn_of<0>(m) : batch_fn_of<1>(m); }

cudaError_t launch_batch_fp64(const FP64BatchArgs &a, int form, int blocks, int threads, cudaStream_t s) {
  void *args[] = {(void *)&a};
  return cudaLaunchKernel(batch_fn(form, store_mode(a.U, a.K, a.V, a.layout)), dim3(blocks), dim3(threads), args, 0, s);
}

int batch_fp64_max_blocks_per_sm(int form, int threads) {
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_fn(form, ST_LANE), threads, 0);
  return (e == cudaSuccess && n > 0) ? n : 1;
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

template <int FORM>
static const void *staged_fn_of(StoreMode m) {
  switch (m) {
    case ST_RING: return (const void *)k_solve_staged<FORM, ST_RING>;
    case ST_PLANES: return (const void *)k_solve_staged<FORM, ST_PLANES>;
    default: return (const void *)k_solve_staged<FORM, ST_LANE>;
  }
}
template <int FORM, bool GREY>
static const void *direct_fn_of(StoreMode m) { /* planes: the lane-by-lane kernel stores no level either */
  return m == ST_RING ? (const void *)k_solve<FORM, GREY, ST_RING> : (const void *)k_solve<FORM, GREY, ST_LANE>;
}
static const void *solve_fn(int form, int grey, bool staged, StoreMode m) {
  if (staged) return form == 0 ? staged_fn_of<0>(m) : staged_fn_of<1>(m);
  if (grey) return form == 0 ? direct_fn_of<0, true>(m) : direct_fn_of<1, true>(m);
  return form == 0 ? direct_fn_of<0, false>(m) : direct_fn_of<1, false>(m);
}

int solve_fp64_max_blocks_per_sm(int form, int grey, int threads) {
  int nb = 0, nb2 = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, solve_fn(form, grey, false, ST_LANE), threads, 0) != cudaSuccess)
    nb = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb2, solve_fn(form, grey, true, ST_LANE), threads, 0) != cudaSuccess)
    nb2 = 1;
  nb = nb > nb2 ? nb : nb2;
  return nb > 0 ? nb : 1;
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

cudaError_t launch_solve_fp64(const SolveArgs &a, int form, int grey, int blocks, int threads, cudaStream_t s) {
  const bool staged = !grey && solve_uses_staging(a.nw);
  void *args[] = {(void *)&a};
  return cudaLaunchKernel(solve_fn(form, grey, staged, store_mode(a.U, a.K, a.V, a.layout)), dim3(blocks), dim3(threads), args, 0, s);
}

}  // namespace oco
