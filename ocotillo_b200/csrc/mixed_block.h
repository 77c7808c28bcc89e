/*
 * mixed_block.h -- what the mixed-precision kernels share besides the arithmetic (mixed_core.h): access to
 * the records, the scratch, the solve of one (column, wavelength) item and the re-solve's lists.
 */
#ifndef OCO_MIXED_BLOCK_H
#define OCO_MIXED_BLOCK_H

#include <cuda_runtime.h>

#include "mixed_core.h"
#include "oco_internal.h"
#include "stores.h"

namespace oco {
using namespace oco::mx;

constexpr int MZC = 14;            /* z records per staged chunk (14 x 256 B) */
constexpr int MWARPS = 4;          /* warps per 128-thread block */
#ifndef MBLOCKS
#define MBLOCKS 5 /* resident blocks per SM */
#endif
constexpr long long kMSpinLimit = 1ll << 26;
constexpr int MG = 4;              /* reverse sweep: levels per group of scratch loads */
constexpr int MIXED_L2_AHEAD = 8;  /* reverse sweep: steps between the L2 prefetch and the load of a level */

/* Shared-memory record accessor. */
struct MRec {
  const float *p;
  __device__ __forceinline__ float operator[](int f) const { return p[f]; }
};
struct MGRec {
  const float *p;
  __device__ __forceinline__ float operator[](int f) const { return __ldg(p + f); }
};

__device__ __forceinline__ uint32_t msmem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mtry_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

/* Per-warp double-buffered stream of one column's records (see StagedPillars in
 * fp64_block.h for the protocol). */
struct MStaged {
  float *buf;
  uint32_t bar0;
  const float *src, *rec; /* the column; the next record in the buffer */
  int nz, nchunks, cur, left;
  uint32_t waits, inflight;
  bool failed;
  __device__ __forceinline__ void issue(int c) {
    const int rows = min(MZC, nz - c * MZC);
    const uint32_t bytes = (uint32_t)(rows * MZN * sizeof(float));
    const uint32_t bar = bar0 + 8u * (c & 1);
    const uint32_t dst = msmem(buf + (c & 1) * (MZC * MZN));
    const size_t g = __cvta_generic_to_global(src + (int64_t)c * MZC * MZN);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(g), "r"(bytes), "r"(bar)
                 : "memory");
  }
  __device__ __forceinline__ bool wait(int b) {
    if (!((inflight >> b) & 1u)) return true;
    const uint32_t bar = bar0 + 8u * b;
    const uint32_t parity = (waits >> b) & 1u;
    long long spins = 0;
    while (!mtry_wait(bar, parity))
      if (++spins > kMSpinLimit) return false;
    waits ^= 1u << b;
    inflight &= ~(1u << b);
    return true;
  }
  __device__ __forceinline__ void begin(const float *column) {
    src = column;
    cur = -1;
    left = 0;
    nchunks = (nz + MZC - 1) / MZC;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); /* this lane's tile accesses before the copies */
    __syncwarp();
    if ((threadIdx.x & 31) == 0) issue(0);
    inflight |= 1u;
  }
  /* The next record; z counts up from 0. */
  __device__ __forceinline__ MRec at(int) {
    if (left == 0) {
      const int c = ++cur;
      __syncwarp();
      if (!failed && c + 1 < nchunks) {
        if ((threadIdx.x & 31) == 0) issue(c + 1);
        inflight |= 1u << ((c + 1) & 1);
      }
      if (!failed && !wait(c & 1)) failed = true;
      rec = buf + (c & 1) * (MZC * MZN);
      left = MZC;
    }
    left--;
    const MRec r{rec};
    rec += MZN;
    return r;
  }
};

struct MDirect {
  const float *base;
  __device__ __forceinline__ MGRec at(int z) { return MGRec{base + (int64_t)z * MZN}; }
};

/* Wavelength constants: most are read only where T changes or at ionized points, so a staged warp
 * keeps them in its shared table [MLN][32] and leaves their registers to the sweep; the lanes of the
 * other kernels hold theirs in registers. */
struct MLamS {
  const float *p; /* &table[0][lane] */
  __device__ __forceinline__ float operator()(int k) const { return p[k * 32]; }
};
__device__ __forceinline__ Lam32 load_lam32(const float *__restrict__ t, int iw, int nw) {
  Lam32 L;
  lam32_from(L, [&](int f) { return __ldg(t + (int64_t)f * nw + iw); });
  return L;
}
__device__ __forceinline__ void store_lam32_shared(float *table, int lane, const float *__restrict__ t, int iw, int nw) {
#pragma unroll
  for (int k = 0; k < MLN; k++) table[k * 32 + lane] = __ldg(t + (int64_t)k * nw + iw);
}

/* Everything one (column, wavelength) item needs besides its records. */
struct MItem {
  const float *lam; /* wavelength table [MLN][nw] of the item's grid */
  int nz, nw, iw;
  float dzf;        /* dz */
  float ldz2i, ldz2f; /* log2(dz^2) = integer + fraction */
  float dz2f;       /* dz^2 */
  double dz1;       /* 1/dz */
  OutPtrs o;        /* U, kappa, V; written only when active */
  double *vtop, *vbot; /* emergent-flux destinations or NULL */
};

/* Item of the block kernels: column cl of the chunk, wavelength iw. */
__device__ __forceinline__ MItem block_item(const MixedArgs &a, int64_t cl, int iw) {
  MItem it;
  it.lam = a.lam;
  it.nz = a.nz;
  it.nw = a.nw;
  it.iw = iw;
  it.dzf = (float)a.dz;
  it.ldz2i = a.ldz2i;
  it.ldz2f = a.ldz2f;
  it.dz2f = (float)(a.dz * a.dz);
  it.dz1 = 1.0 / a.dz;
  const int64_t idx = (a.layout == 0) ? (int64_t)iw * a.ld_col + a.c_off + cl : (a.c_off + cl) * a.nw + iw;
  it.o.U = a.U ? a.U + idx * a.U_is : nullptr;
  it.o.K = a.K ? a.K + idx * a.K_is : nullptr;
  it.o.V = a.V ? a.V + idx * a.V_is : nullptr;
  it.o.uz = a.U_zs;
  it.o.kz = a.K_zs;
  it.o.vz = a.V_zs;
  it.o.urow = a.ld_col * a.U_is;
  it.o.krow = a.ld_col * (int64_t)a.nz;
  const int64_t pidx = (int64_t)iw * a.ld_col + a.c_off + cl;
  it.vtop = a.Vtop ? a.Vtop + pidx : nullptr;
  it.vbot = a.Vbot ? a.Vbot + pidx : nullptr;
  return it;
}

/* The warp's Thomas scratch, one sequential stream per warp.  A record per level is
 * {v, kappa or 1/kappa, u mantissa, u exponent} (see the forward sweep); two formats:
 *   MScratch16  one float4 per lane, 512 bytes per level;
 *   MScratch12  12 bytes per lane, 384 per level: the 32 lanes' {v, kappa} pairs (float2),
 *               then their u mantissas, with u's exponent packed into the spare bits of kappa
 *               and of the mantissa (pack_o1_u, mixed_core.h: u's mantissa lies in [1, 2)).  A
 *               record whose u does not fit (exponent outside [-512, 511], or a mantissa that
 *               is not normal) makes put() return false and the item is flagged for the FP64
 *               re-solve (on the AGN and Athena-style grids the exponent stays in [-420, 90]).
 * Both store the same values, so the results are the same bits.  The 12-byte records move a
 * quarter less scratch for ~4% more instructions: the ragged batches (longest columns first, up
 * to 2048 levels) use them (c4 batch 25.0 -> 23.7 ms), the block solves keep float4 records
 * (12-byte records measured 0.7% slower on the 512-level AGN grid, 2% on the 1024-level
 * precision grid). */
struct MScratch16 {
  static constexpr int LEVEL = 32 * 16;
  char *w; /* the warp's level 0 */
  int lane;
  __device__ __forceinline__ float4 *p(int j) const { return (float4 *)(w + (int64_t)j * LEVEL) + lane; }
  __device__ __forceinline__ const char *level(int j) const { return w + (int64_t)j * LEVEL; }
  __device__ __forceinline__ bool put(int j, const float4 &r) const {
    *p(j) = r;
    return true;
  }
  using Raw = float4; /* a record as loaded; opened where it is used, so that the load stays in flight */
  __device__ __forceinline__ Raw load(int j) const { return *p(j); }
  static __device__ __forceinline__ float4 open(const Raw &r) { return r; }
  __device__ __forceinline__ float4 get(int j) const { return *p(j); }
  __device__ __forceinline__ float kappa(int j) const { return p(j)->y; }
};
struct MScratch12 {
  static constexpr int LEVEL = 32 * 12;
  char *w; /* the warp's level 0 */
  int lane;
  __device__ __forceinline__ float2 *p2(int j) const { return (float2 *)(w + (int64_t)j * LEVEL) + lane; }
  __device__ __forceinline__ float *p1(int j) const { return (float *)(w + (int64_t)j * LEVEL + 256) + lane; }
  __device__ __forceinline__ const char *level(int j) const { return w + (int64_t)j * LEVEL; }
  __device__ __forceinline__ bool put(int j, const float4 &r) const {
    int w1, w2;
    const bool fits = pack_o1_u(r.y, r.z, __float_as_int(r.w), w1, w2);
    *p2(j) = make_float2(r.x, __int_as_float(w1));
    *p1(j) = __int_as_float(w2);
    return fits;
  }
  struct Raw {
    float2 a;
    float m;
  };
  __device__ __forceinline__ Raw load(int j) const { return Raw{*p2(j), *p1(j)}; }
  static __device__ __forceinline__ float4 open(const Raw &r) {
    float kc, m;
    int e;
    unpack_o1_u(__float_as_int(r.a.y), __float_as_int(r.m), kc, m, e);
    return make_float4(r.a.x, kc, m, __int_as_float(e));
  }
  __device__ __forceinline__ float4 get(int j) const { return open(load(j)); }
  __device__ __forceinline__ float kappa(int j) const { return __int_as_float(__float_as_int(p2(j)->y) & 0x7fffffff); }
};
/* MScratch12P: 12 bytes without kappa, for solves that store no level (the kappa of the two ends stays
 * with the item): {v, u mantissa} (float2), then u's exponents; no packing, any exponent. */
struct MScratch12P {
  static constexpr int LEVEL = 32 * 12;
  char *w; /* the warp's level 0 */
  int lane;
  __device__ __forceinline__ float2 *p2(int j) const { return (float2 *)(w + (int64_t)j * LEVEL) + lane; }
  __device__ __forceinline__ float *p1(int j) const { return (float *)(w + (int64_t)j * LEVEL + 256) + lane; }
  __device__ __forceinline__ const char *level(int j) const { return w + (int64_t)j * LEVEL; }
  __device__ __forceinline__ bool put(int j, const float4 &r) const {
    *p2(j) = make_float2(r.x, r.z);
    *p1(j) = r.w;
    return true;
  }
  struct Raw {
    float2 a;
    float e;
  };
  __device__ __forceinline__ Raw load(int j) const { return Raw{*p2(j), *p1(j)}; }
  static __device__ __forceinline__ float4 open(const Raw &r) { return make_float4(r.a.x, 0.0f, r.a.y, r.e); }
  __device__ __forceinline__ float4 get(int j) const { return open(load(j)); }
  __device__ __forceinline__ float kappa(int) const { return 0.0f; } /* not kept */
};
/* One (column, wavelength) item, its scratch records in sc.  An inactive lane runs the forward
 * sweep (to keep a staged warp in step) and writes nothing. */
/* Returns whether the item's emergent flux is ill-conditioned for this arithmetic: with
 * D_k = u_k - q_k U_{k+1} (all three terms >= 0) and the boundary flux proportional to
 * 37 D_a - 8 D_b + D_c (the 6th-order stencil with mirrored ghost differences; a, b, c the
 * three differences next to the boundary), its condition number with respect to relative
 * errors of u, q and U is
 *   (37 C_a + 8 C_b + C_c) / |37 D_a - 8 D_b + D_c|,   C_k = u_k + q_k U_{k+1};
 * FP32 leaves relative errors of a few 1e-6 in u, q and U, so above `cond` the item is
 * flagged for the FP64 re-solve (kernels_repair.cu).  Columns with nz < 4 are not tested (their flux is the
 * reference's stencil on U).  An item whose scratch records do not fit MScratch is flagged too. */
template <class PA, class LA, class SC, class ST>
__device__ __forceinline__ bool msolve_item(const MItem &it, bool active, PA &pa, const LA &L, const SC &sc,
                                            ST st, float cond) {
  const int nz = it.nz;
  const float dzf = it.dzf, dz2f = it.dz2f, ldz2i = it.ldz2i, ldz2f = it.ldz2f;

  /* The (T, lambda) part is taken again while the record says that T has not changed: most levels
   * of a disk sit at its temperature floor.  356 -> 300 instructions per point on the AGN grid
   * (4096 columns x 512 x 256, all of the kernel: 6.77 -> 6.1 ms). */
  const LamPt c = lam_point(L);
  TF32 t;
  auto opac = [&](int z) -> Opac32 {
    const auto Z = pa.at(z);
    if (!(f2bits(Z[MZ_FLAGS]) & MZF_SAME_T)) t = tfac(Z, L);
    return opacity(Z, L, c, t);
  };
  Opac32 cur = opac(0);
  Opac32 nxt = opac(1);
  float kc = kappa_lin(cur), kn = kappa_lin(nxt);
  const float k0 = kc; /* kappa of the bottom level */
  /* What a level's scratch record keeps of kappa: kappa itself where it leaves in the reverse sweep (the
   * ring), else 1/kappa, which is all that the fluxes need then: kappa is stored by the forward sweep,
   * and the reverse sweep, the longer chain, has no reciprocal, conversion and third store (ragged batch of
   * 8192 columns 24.0 -> 22.1 ms, AGN grid of 4096 columns 6.60 -> 6.32 ms). */
  constexpr bool KREV = ST::KAPPA_REVERSE;
  auto keep = [](float k) -> float { return KREV || ST::PLANES ? k : rcp(k); };
  auto kept_o1 = [](float y) -> float { return KREV || ST::PLANES ? rcp(y) : y; };
  if (!KREV) st.k(0, (double)kc);
  Row32 r = row_boundary(kc, cur, dzf, dz2f, ldz2i, ldz2f, false);
  float h = r.e, cprev = r.c;
  float an = 2.0f * rcp(kn + kc); /* a' of row 1; then c' of the row below */
  XF u = xexp2(r.ldi, r.ldf);
  u = xnorm(u.m * (r.w * rcp(r.c + h)), u.e);
  /* scratch record of z = j: {v_j, keep(kappa_j), u_j mantissa, u_j exponent (int bits)} where v_j holds the
   * smaller of q_j = h_j/(c_j+h_j) and |gamma_{j+1}| = c_j/(c_j+h_j) (they sum to 1; a negative
   * v_j stores -|gamma_{j+1}|), written once row j+1 is known */
  float4 pend = make_float4(0.0f, keep(kc), u.m, __int_as_float(u.e));
  bool fits = true;
  for (int j = 1; j < nz; j++) {
    cur = nxt;
    kc = kn;
    if (j < nz - 1) {
      nxt = opac(j + 1);
      kn = kappa_lin(nxt);
      r = row_center(an, kc, kn, cur, dz2f, ldz2i, ldz2f);
      an = r.c;
    } else {
      r = row_boundary(kc, cur, dzf, dz2f, ldz2i, ldz2f, true);
    }
    const float rr = rcp(cprev + h);
    const float qv = h * rr, gv = cprev * rr;
    pend.x = (qv < gv) ? qv : -gv;
    fits &= sc.put(j - 1, pend);
    h = r.e + (r.a * rr) * h; /* a'/(c'+h) is O(1); a' h alone can overflow */
    const float rb = rcp(r.c + h);
    u = xaxpy(xexp2(r.ldi, r.ldf), r.w * rb, u, r.a * rb);
    pend = make_float4(0.0f, keep(kc), u.m, __int_as_float(u.e));
    if (!KREV) st.k(j, (double)kc);
    cprev = r.c;
  }
  fits &= sc.put(nz - 1, pend);
  bool flag = !fits;

  /* reverse sweep */
  const int n = nz;
  const double dz1 = it.dz1;
  XF Un = u; /* U_{n-1} */
  double vtop = 0.0, vbot = 0.0;
  if (nz >= 4) {
    st.open(n);
    st.push_u(3, n + 2, xtod(Un));
    /* window of differences d0..d5 = D_k..D_{k+5}; V_{k+3} from it */
    double d0, d1, d2, d3, d4, d5;
    double Uk[3];
    /* D_{n-2}, D_{n-3}, D_{n-4} first (top ghosts mirror them) */
    double Dt[3];
    float kt[3];
    double Ct[3]; /* C_k = u_k + q_k U_{k+1} of the top differences */
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const int k = n - 2 - t;
      const float4 w = sc.get(k);
      kt[t] = w.y;
      const float g1 = (w.x >= 0.0f) ? 1.0f - w.x : -w.x;
      const float qk = (w.x >= 0.0f) ? w.x : 1.0f + w.x;
      XF uj;
      uj.m = w.z;
      uj.e = __float_as_int(w.w);
      const double Uk1 = t == 0 ? xtod(Un) : Uk[t - 1];
      Ct[t] = xtod(uj) + (double)qk * Uk1;
      XF Dj;
      xaxpy2(uj, Un, g1, -qk, Un, Dj);
      Uk[t] = xtod(Un);
      if (t < 2) st.push_u(4 + t, 3 + k, Uk[t]);
      Dt[t] = xtod(Dj);
    }
    flag = flag || !(37.0 * Ct[0] + 8.0 * Ct[1] + Ct[2] <= (double)cond * fabs(37.0 * Dt[0] - 8.0 * Dt[1] + Dt[2]));
    /* top ghosts f(n2+i) = 2 f(n2) - f(n2-i) */
    const double fn = xtod(u);
    st.push_u(2, n + 3, 2.0 * fn - Uk[0]);
    st.push_u(1, n + 4, 2.0 * fn - Uk[1]);
    st.push_u(0, n + 5, 2.0 * fn - Uk[2]);
    /* window for V_{n-1}: D_{n-4} .. D_{n+1} = Dt[2], Dt[1], Dt[0], D_{n-1}=Dt[0], D_n=Dt[1], D_{n+1}=Dt[2] */
    d0 = Dt[2]; d1 = Dt[1]; d2 = Dt[0]; d3 = Dt[0]; d4 = Dt[1]; d5 = Dt[2];
    auto flux = [&](float kj) -> double {
      const double s1 = d2 + d3;
      const double s2 = (s1 + d1) + d4;
      const double s3 = (s2 + d0) + d5;
      const double df = -((1.0 / 60.0) * (((45.0 * s1) - 9.0 * s2) + s3));
      return ((-(double)kept_o1(kj)) * df) * dz1;
    };
    {
      const float kj = keep(kc); /* the top level's */
      vtop = flux(kj);
      st.push(6, n - 1, Uk[2], vtop, (double)kj); /* U_{n-4}, V_{n-1} */
      st.template group<false>(n - 1, 7);
    }
    double U0 = Uk[2], U1 = Uk[1], U2 = Uk[0], U3 = fn; /* the four lowest U seen so far */
    /* r1, r2, r3 = what the records keep of kappa of k+1, k+2, k+3 before step k */
    float r1 = kt[2], r2 = kt[1], r3 = kt[0];
    auto step = [&](int slot, int k, const float4 &w) {
      const float g1 = (w.x >= 0.0f) ? 1.0f - w.x : -w.x; /* |gamma_{k+1}| */
      const float qk = (w.x >= 0.0f) ? w.x : 1.0f + w.x;  /* q_k */
      XF uj;
      uj.m = w.z;
      uj.e = __float_as_int(w.w);
      XF Dj;
      xaxpy2(uj, Un, g1, -qk, Un, Dj);
      const double Uv = xtod(Un);
      U3 = U2; U2 = U1; U1 = U0; U0 = Uv;
      d5 = d4; d4 = d3; d3 = d2; d2 = d1; d1 = d0; d0 = xtod(Dj);
      st.push(slot, 3 + k, Uv, flux(r3), (double)r3);
      r3 = r2; r2 = r1; r1 = w.y;
    };
    int k = n - 5;
    /* Scratch levels in two groups of MG that take turns (one in use, one in flight); one bulk request
     * from lane 0 brings the MG levels MIXED_L2_AHEAD steps further down into L2 (the warp's levels
     * are contiguous; they were written a whole forward sweep ago and have usually left L2). */
    if (k >= 7 + (ST::PLANES ? 4 : 0)) {
      typename SC::Raw A[MG], B[MG];
      auto load = [&](typename SC::Raw *w, int k0) {
        if (k0 - MG + 1 - MIXED_L2_AHEAD >= 0 && (threadIdx.x & 31) == 0)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(
                           sc.level(k0 - MG + 1 - MIXED_L2_AHEAD))),
                       "r"((uint32_t)(MG * SC::LEVEL))
                       : "memory");
#pragma unroll
        for (int i = 0; i < MG; i++) w[i] = sc.load(max(k0 - i, 0));
      };
      auto steps = [&](const typename SC::Raw *w, int slot, int k0) {
#pragma unroll
        for (int i = 0; i < MG; i++) {
          const float4 x = SC::open(w[i]);
          if constexpr (ST::PLANES) { /* U alone down to the bottom's last levels */
            const XF uj{x.z, __float_as_int(x.w)};
            Un = xaxpy1(uj, Un, (x.x >= 0.0f) ? 1.0f - x.x : -x.x);
          } else {
            step(slot + i, k0 - i, x);
          }
        }
      };
      load(A, k);
      for (; k >= 7 + (ST::PLANES ? 4 : 0); k -= 8) {
        load(B, k - MG);
        steps(A, 0, k);
        load(A, k - 8);
        steps(B, MG, k - MG);
        st.template group<true>(3 + k - 7, 8);
      }
    }
    int q = 0;
#pragma unroll 1
    for (; k >= 0; k--) {
      step(q, k, sc.get(k));
      if (++q == 8) {
        st.template group<false>(3 + k, 8);
        q = 0;
      }
    }
    { /* condition number of the bottom flux from D_0, D_1, D_2 (d0, d1, d2) and U_1..U_3 */
      double Cb = 0.0;
#pragma unroll
      for (int t = 0; t < 3; t++) {
        const float4 w = sc.get(t);
        const float qk = (w.x >= 0.0f) ? w.x : 1.0f + w.x;
        XF uj;
        uj.m = w.z;
        uj.e = __float_as_int(w.w);
        const double Ck = xtod(uj) + (double)qk * (t == 0 ? U1 : (t == 1 ? U2 : U3));
        Cb += (t == 0 ? 37.0 : (t == 1 ? 8.0 : 1.0)) * Ck;
      }
      flag = flag || !(Cb <= (double)cond * fabs(37.0 * d0 - 8.0 * d1 + d2));
    }
    /* bottom ghosts f(n1-i) = 2 f(n1) - f(n1+i); ghost differences mirror D_0, D_1, D_2 */
    const double g0 = 2.0 * U0 - U3, g1 = 2.0 * U0 - U2, g2 = 2.0 * U0 - U1, D0 = d0, D1 = d1, D2 = d2;
#pragma unroll 1
    for (int j = 2; j >= 0; j--) { /* D_{-1} = D_0, D_{-2} = D_1, D_{-3} = D_2 */
      d5 = d4; d4 = d3; d3 = d2; d2 = d1; d1 = d0; d0 = j == 2 ? D0 : (j == 1 ? D1 : D2);
      const float kj = ST::PLANES ? k0 : j == 2 ? r3 : (j == 1 ? r2 : r1);
      vbot = flux(kj);
      st.push(q, j, j == 2 ? g2 : (j == 1 ? g1 : g0), vbot, (double)kj);
      if (++q == 8) {
        st.template group<false>(j, 8);
        q = 0;
      }
    }
    st.finish(q);
  } else { /* nz = 2 or 3: U stencil on the ghosted array (the reference's update order) */
    double f[9];
    const int n1 = 3, n2 = nz + 2;
    f[n1 + nz - 1] = xtod(Un);
    for (int j = nz - 2; j >= 0; j--) {
      const float4 w = sc.get(j);
      const float g1 = (w.x >= 0.0f) ? 1.0f - w.x : -w.x;
      XF uj;
      uj.m = w.z;
      uj.e = __float_as_int(w.w);
      XF Dj;
      xaxpy2(uj, Un, g1, 0.0f, Un, Dj);
      f[n1 + j] = xtod(Un);
    }
    for (int i = 1; i <= 3; i++) {
      f[n1 - i] = 2.0 * f[n1] - f[n1 + i];
      f[n2 + i] = 2.0 * f[n2] - f[n2 - i];
    }
    for (int m = 0; m < nz + 6; m++) st.u(m, f[m]);
    for (int j = 0; j < nz; j++) {
      const int c = n1 + j;
      const double df = (1.0 / 60.0) * (((45.0 * (f[c + 1] - f[c - 1])) - 9.0 * (f[c + 2] - f[c - 2])) + (f[c + 3] - f[c - 3]));
      const float kj = ST::PLANES ? (j == 0 ? k0 : kc) : sc.kappa(j);
      const double v = ((-(double)kept_o1(kj)) * df) * dz1;
      st.v(j, v);
      if (KREV) st.k(j, (double)kj);
      if (j == 0) vbot = v;
      if (j == nz - 1) vtop = v;
    }
  }
  if (!active) return false;
  if (it.vtop) __stcs(it.vtop, vtop);
  if (it.vbot) __stcs(it.vbot, vbot);
  return flag;
}

/* The re-solve's lists (RepairArgs): each flagged item's id goes to ilist (its index there is
 * the item's slot, also stored beside its bit), and each word of flag bits (a column's 32
 * wavelengths) that receives a bit goes to wlist once.  mark_tile serves the tilings whose warp
 * task is one (column, 32-wavelength tile): the tile is one word and no other warp writes it, so
 * lane 0 stores the warp's ballot.  mark_items serves the tilings whose 32 items may span
 * columns: each flagged lane sets its bit, and the lane that finds its word empty lists it. */
__device__ __forceinline__ void list_items(bool flag, unsigned m, unsigned long long id, int64_t word, int iw,
                                           unsigned long long *ilist, unsigned long long *icount, int *slot) {
  const int lane = threadIdx.x & 31, first = __ffs(m) - 1;
  unsigned long long base = 0;
  if (lane == first) base = atomicAdd(icount, (unsigned long long)__popc(m));
  base = __shfl_sync(0xffffffffu, base, first);
  if (flag) {
    const unsigned long long pos = base + __popc(m & ((1u << lane) - 1u));
    ilist[pos] = id;
    slot[word * 32 + (iw & 31)] = (int)pos;
  }
}

__device__ __forceinline__ void mark_tile(bool flag, int64_t word, int iw, unsigned long long id, unsigned *bits,
                                          int *slot, unsigned long long *wlist, unsigned long long *wcount,
                                          unsigned long long *ilist, unsigned long long *icount) {
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  if (!m) return;
  if ((threadIdx.x & 31) == 0) {
    bits[word] = m;
    wlist[atomicAdd(wcount, 1ull)] = (unsigned long long)word;
  }
  list_items(flag, m, id, word, iw, ilist, icount, slot);
}

__device__ __forceinline__ void mark_items(bool flag, int64_t word, int iw, unsigned long long id, unsigned *bits,
                                           int *slot, unsigned long long *wlist, unsigned long long *wcount,
                                           unsigned long long *ilist, unsigned long long *icount) {
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  if (!m) return;
  if (flag && atomicOr(bits + word, 1u << (iw & 31)) == 0u) wlist[atomicAdd(wcount, 1ull)] = (unsigned long long)word;
  list_items(flag, m, id, word, iw, ilist, icount, slot);
}

/* A staged warp's shared memory; the output ring of the reverse sweep takes over what the forward
 * sweep used (the next task rewrites it; see MStaged::begin). */
struct MStagedSmem {
  union {
    struct {
      float rec[2 * MZC * MZN];
      float lam[MLN * 32]; /* the task's 32 wavelengths' constants */
    };
    RingSmem<float> ring;
  };
  unsigned long long bar[2];
  __device__ MStagedSmem() = delete;
};
static_assert(sizeof(MStagedSmem) % 16 == 0, "bulk copies");

__device__ __forceinline__ void init_staged(MStaged &pa, MStagedSmem &sm) {
  pa.buf = sm.rec;
  pa.bar0 = msmem(&sm.bar[0]);
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

#endif /* OCO_MIXED_BLOCK_H */
