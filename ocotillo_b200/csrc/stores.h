/*
 * stores.h -- where the reverse sweeps' outputs go (FP64 and mixed kernels).
 *
 * The sweeps hand over the levels m = nz + 5 .. 0 of U's ghosted index in decreasing order, with V
 * and kappa of interior level m where there is one (m < nz): a first group of 7 levels (the top
 * ghosts and the four uppermost levels), then groups of 8.
 *
 * LaneStores: each lane writes its item's levels itself (coalesced where lambda is the fastest
 * index).
 *
 * RingStores, for layouts with z fastest (the reference's): neighbouring lanes' levels lie a row
 * apart, so the levels go through a ring of 15 in shared memory, and each group of 8 lets every
 * row write one run of 8 that starts on a 64-byte boundary of its own (rows of nz or nz + 6
 * elements start anywhere), four rows per store instruction.  Runs at the same level in every row
 * leave partial sectors, which L2 cannot keep until the next group completes them once three
 * arrays are written (AGN grid of 1600 columns, mixed: 6.3 ms so, 3.2 ms with one array; 3.43 ms
 * with the runs on boundaries; lambda-fastest temporaries and three transposes 5.0 ms).
 * ROWS: the warp's rows are equally spaced (one column's wavelengths), otherwise each row's
 * address comes from its lane.  Every lane of the warp takes part with the same number of levels;
 * the active ones come first.
 */
#ifndef OCO_STORES_H
#define OCO_STORES_H

#include <cstdint>

#include <cuda_runtime.h>

#include "oco_internal.h"

namespace oco {

struct OutPtrs {
  double *U, *K, *V;     /* z = 0 (U: ghost zone 0) or NULL */
  int64_t uz, kz, vz;    /* strides between levels */
  int64_t urow, krow;    /* z fastest: elements between the rows of neighbouring wavelengths */
};

/* KREV: kappa leaves with U and V in the reverse sweep (push's last argument), otherwise the
 * forward sweep has stored it (k) and the argument is ignored. */
template <bool KREV>
struct LaneStores {
  static constexpr bool KAPPA_REVERSE = KREV, PLANES = false;
  double *Ub, *Kb, *Vb;
  int64_t uz, kz, vz;
  __device__ __forceinline__ LaneStores(const OutPtrs &o, bool active)
      : Ub(active ? o.U : nullptr), Kb(active ? o.K : nullptr), Vb(active ? o.V : nullptr), uz(o.uz), kz(o.kz),
        vz(o.vz) {}
  __device__ __forceinline__ void u(int m, double x) const {
    if (Ub) __stcs(&Ub[m * uz], x);
  }
  __device__ __forceinline__ void k(int j, double x) const {
    if (Kb) __stcs(&Kb[j * kz], x);
  }
  __device__ __forceinline__ void v(int j, double x) const {
    if (Vb) __stcs(&Vb[j * vz], x);
  }
  __device__ __forceinline__ void open(int) {}
  __device__ __forceinline__ void push_u(int, int m, double U) { u(m, U); }
  __device__ __forceinline__ void push(int, int m, double U, double V, double K) {
    u(m, U);
    v(m, V);
    if (KREV) k(m, K);
  }
  template <bool FULL>
  __device__ __forceinline__ void group(int, int) {}
  __device__ __forceinline__ void finish(int) {}
};

/* Only the emergent planes are wanted (a serving job without fields): nothing is stored per level.
 * The sweeps then form the fluxes and differences of the bottom levels alone, and the scratch keeps
 * kappa of the two ends only. */
struct PlaneStores {
  static constexpr bool KAPPA_REVERSE = false, PLANES = true;
  __device__ __forceinline__ void u(int, double) const {}
  __device__ __forceinline__ void k(int, double) const {}
  __device__ __forceinline__ void v(int, double) const {}
  __device__ __forceinline__ void open(int) {}
  __device__ __forceinline__ void push_u(int, int, double) {}
  __device__ __forceinline__ void push(int, int, double, double, double) {}
  template <bool FULL>
  __device__ __forceinline__ void group(int, int) {}
  __device__ __forceinline__ void finish(int) {}
};

constexpr int RING_Z = 15, RING_ROW = 33; /* 33: conflict-free both ways */
/* KT: type that holds kappa exactly (float in the mixed form). */
template <class KT>
struct RingSmem {
  double U[RING_Z * RING_ROW], V[RING_Z * RING_ROW];
  KT K[RING_Z * RING_ROW];
};

template <bool ROWS, class KT>
struct RingStores : LaneStores<true> { /* the base's stores serve columns of fewer than 4 levels */
  RingSmem<KT> *ring;
  double *U0, *K0, *V0; /* row of lane / 8 (ROWS) or of the lane */
  int64_t us, ks;       /* elements between rows */
  int nz, nrows, base;  /* base: ring slot of the group's first level */
  __device__ __forceinline__ RingStores(const OutPtrs &o, bool active, RingSmem<KT> *r)
      : LaneStores<true>(o, active), ring(r), U0(o.U), K0(o.K), V0(o.V), us(o.urow), ks(o.krow), nz(0), base(0) {
    nrows = __popc(__ballot_sync(0xffffffffu, active)); /* active lanes come first */
    if (ROWS) {
      const int r8 = (threadIdx.x & 31) / 8;
      U0 = (double *)__shfl_sync(0xffffffffu, (unsigned long long)U0, 0);
      K0 = (double *)__shfl_sync(0xffffffffu, (unsigned long long)K0, 0);
      V0 = (double *)__shfl_sync(0xffffffffu, (unsigned long long)V0, 0);
      if (U0) U0 += r8 * us;
      if (K0) K0 += r8 * ks;
      if (V0) V0 += r8 * ks;
    }
  }
  /* Before an item's first push.  The ring may lie over shared memory that the forward sweep read
   * (StagedSmem, MStagedSmem): no lane writes it before every lane has left that sweep. */
  __device__ __forceinline__ void open(int n) {
    nz = n;
    base = 0;
    __syncwarp();
  }
  static __device__ __forceinline__ int wrap(int s) { return s >= RING_Z ? s - RING_Z : s; }
  /* level m, the q-th of its group */
  __device__ __forceinline__ void push_u(int q, int, double U) { ring->U[wrap(base + q) * RING_ROW + (threadIdx.x & 31)] = U; }
  __device__ __forceinline__ void push(int q, int, double U, double V, double K) {
    const int i = wrap(base + q) * RING_ROW + (threadIdx.x & 31);
    ring->U[i] = U;
    ring->V[i] = V;
    ring->K[i] = (KT)K;
  }
  /* One array's runs after every level above lo (ring slot slo) has been pushed: row r, whose
   * element 0 lies ph elements past a 64-byte boundary, writes levels w .. w + 7 with w the lowest
   * level >= lo on a boundary.  top: levels above are not stored; full: all 8 levels of every
   * row are. */
  template <class T>
  __device__ __forceinline__ void runs(const T *a, double *p, int64_t stride, int lo, int slo, int top, bool full) const {
    if (!p) return;
    const int lane = threadIdx.x & 31, s = lane & 7, r = lane / 8;
    if (ROWS) {
      const int w = (int)(-((int64_t)((unsigned long long)p >> 3) + lo)) & 7;
      /* rows 4 apart: 4 stride elements, 0 or 4 past a boundary */
      const int oe = w + s, oo = ((w + ((int)(stride & 1) << 2)) & 7) + s;
      const T *ae = a + (slo - oe + (slo < oe ? RING_Z : 0)) * RING_ROW + r;
      const T *ao = a + (slo - oo + (slo < oo ? RING_Z : 0)) * RING_ROW + r;
      double *ge = p + lo + oe, *go = p + lo + oo;
      if (full) {
#pragma unroll
        for (int i = 0; i < 8; i++) ((i & 1) ? go : ge)[(int64_t)(4 * i) * stride] = (double)((i & 1) ? ao : ae)[4 * i];
      } else {
        const bool one = lo + oe <= top && lo + oe >= 0, two = lo + oo <= top && lo + oo >= 0;
#pragma unroll 1
        for (int i = 0; i < 8; i++)
          if (4 * i + r < nrows && ((i & 1) ? two : one))
            ((i & 1) ? go : ge)[(int64_t)(4 * i) * stride] = (double)((i & 1) ? ao : ae)[4 * i];
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < 8; i++) {
        double *q = (double *)__shfl_sync(0xffffffffu, (unsigned long long)p, 4 * i + r);
        const int o = ((int)(-((int64_t)((unsigned long long)q >> 3) + lo)) & 7) + s, m = lo + o;
        if (4 * i + r < nrows && m <= top && m >= 0)
          q[m] = (double)a[(slo - o + (slo < o ? RING_Z : 0)) * RING_ROW + r + 4 * i];
      }
    }
  }
  /* a group of n levels, the lowest lo, is complete; FULL: worth the straight-line code for runs
   * without masks (the main loop's) */
  template <bool FULL>
  __device__ __forceinline__ void group(int lo, int n) {
    const int slo = wrap(base + n - 1);
    const bool full = FULL && lo <= nz - 17 && nrows == 32;
    __syncwarp();
    runs(ring->U, U0, us, lo, slo, nz + 5, full);
    runs(ring->V, V0, ks, lo, slo, nz - 1, full);
    runs(ring->K, K0, ks, lo, slo, nz - 1, full);
    __syncwarp();
    base = wrap(base + n);
  }
  /* level 0 was the q-th level (from 1) of its group, or q = 0: no group open */
  __device__ __forceinline__ void finish(int q) {
#pragma unroll 1
    for (int t = 0; t < 2; t++) group<false>(q - 8 - 8 * t, 8);
  }
};

/* The stores of a StoreMode. */
template <int MODE, bool ROWS, bool KREV, class KT>
__device__ __forceinline__ auto make_stores(const OutPtrs &o, bool active, RingSmem<KT> *ring) {
  if constexpr (MODE == ST_RING)
    return RingStores<ROWS, KT>(o, active, ring);
  else if constexpr (MODE == ST_PLANES)
    return PlaneStores{};
  else
    return LaneStores<KREV>(o, active);
}

}  // namespace oco

#endif /* OCO_STORES_H */
