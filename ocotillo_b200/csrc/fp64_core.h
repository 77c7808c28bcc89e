/*
 * fp64_core.h -- the FP64 per-item arithmetic of the plain and stable forms, shared by the
 * FP64 kernels (kernels_fp64*.cu) and the mixed kernels' FP64 re-solve of flagged items
 * (kernels_mixed.cu).
 *
 *   pillar_record  one (column, z) record: Saha ionization and every factor of the
 *                  reference's per-(z, lambda) opacity that depends on z only
 *                  (gas_state.f90:30-110, continuous_opacity.f90:143-163 and the z-only parts
 *                  of :203-300), each with the reference's operand order.
 *   opacity_at     calc_opacity_and_albedo for one (z, lambda), continuous_opacity.f90:175-201.
 *   solve_item     one (column, wavelength) item: coefficients (auxiliary.f90:111-201), the
 *                  Thomas sweep (:14-47) with its scratch, ghosts (:49-62) and flux (:64-109).
 *
 * Bit-faithfulness to the CPU oracle needs this code compiled without FMA contraction
 * (their units are built with -fmad=false); the exponentials and logarithms (ocomath) use
 * non-contracting intrinsics everywhere.
 */
#ifndef OCO_FP64_CORE_H
#define OCO_FP64_CORE_H

#include <cuda_runtime.h>

#include "ocomath.h"
#include "oco_consts.h"
#include "oco_internal.h"
#include "recip_div.h"
#include "stores.h"

namespace oco {
using namespace k;

/* ---- pillars ------------------------------------------------------------------------ */
/* The record of one (column, z) cell from its rho and T; same_T: the level below it in the column
 * has the same temperature, bit for bit. */
__device__ __forceinline__ void pillar_record(const double r, const double t, double fully_ionized_T, int grey,
                                              bool same_T, double *__restrict__ o) {
  if (grey) { /* grey_parameters, continuous_opacity.f90:383-384 */
    double t2 = t * t;
    o[G_RHO] = r;
    o[G_S] = sigma_sb * (t2 * t2);
    o[G_ALPHA] = (3.68e22 * oco_pow(t, -3.5)) * r;
    return;
  }
  const double rho1 = 1.0 / r; /* gas_state.f90:34-35 */
  const double T1 = 1.0 / t;
  /* calc_hydrogen_ion_frac, gas_state.f90:57-74 */
  double constants = saha_const * oco_pow(t, 1.5);
  double exparg = (T1 * hydrogen_ionization_eV) * k1_eV;
  double niine_ni = constants * oco_exp(-exparg);
  double c_ion = (mp * rho1) * niine_ni;
  double x = 0.5 * (sqrt(c_ion * c_ion + 4.0 * c_ion) - c_ion);
  if (t > fully_ionized_T) x = 1.0;
  /* solve_gas_state, gas_state.f90:85-97 */
  double nn = r * mp1;
  double invn = rho1 * mp;
  double nHII = x * nn;
  double nHI = nn - nHII;
  double ne = nHII;
  double ionf = (nHI != 0.0) ? nHI / (nHI + nHII) : 0.0;
  double Pe = (ne * k_cgs) * t;                    /* gas_state.f90:108 */
  double escat = (alpha_e * nHII) * invn;          /* c_o :149 */
  double theta = 5040.0 * T1;                      /* gas_state.f90:40-43 */
  double theta1 = 1.0 / theta;
  double lgt = oco_log10(theta);
  double hmbf = ((4.158e-10 * Pe) * oco_pow(theta, 2.5)) * oco_pow10(0.754 * theta); /* c_o :161 */
  /* z-only factors of get_kappa_H_bf, c_o :234-242.  chi_n(n) = Ry*(1 - 1*(1/n)**2) as
   * in pre_calc_opacity_quantities :121-129; chi_m equals chi_n(6). */
  double ktemp = k_cgs * t, ktemp1 = k1_cgs * T1;
  double E[6];
#pragma unroll
  for (int nq = 1; nq <= 6; nq++) {
    double n1 = 1.0 / (double)nq;
    double chi_n = RydbergEnergy * (1.0 - 1.0 * (n1 * n1));
    E[nq - 1] = oco_exp(-(chi_n * ktemp1));
  }
  double unsold = ((0.5 * ktemp) * RydbergEnergy1) * (E[5] - oco_exp(-(RydbergEnergy * ktemp1)));
  o[F_RHO] = r;
  o[F_RHO1] = rho1;
  o[F_T1] = T1;
  o[F_DFT1] = damping_factor_const * T1;
  o[F_THETA] = theta;
  o[F_TH1L] = theta1 * log10e;
  o[F_LGT] = lgt;
  o[F_LGT2] = lgt * lgt;
  o[F_IONF] = ionf;
  o[F_ESCAT] = escat;
  o[F_ESCM] = escat * mp1;
  o[F_HMBF] = hmbf;
  o[F_FLAGS] = __hiloint2double(0, (((1.0 - x) > switch_ionfraction) ? FLAG_NEUTRAL : 0) | (same_T ? FLAG_SAME_T : 0) |
                                       (div_a_ok(o[F_ESCM]) ? FLAG_ESC_OK : 0));
#pragma unroll
  for (int q = 0; q < 6; q++) o[F_E1 + q] = E[q];
  o[F_UNSOLD] = unsold;
  o[F_AFF] = ((ionf * ne) * k_cgs) * t;                                             /* c_o :339 */
  o[F_EF] = (((0.5 * log10e) * theta1) * Iev1) * oco_pow10(-(theta * Iev));   /* c_o :265 */
  o[F_TPOW] = oco_pow(t * 1e-4, -1.5);                                              /* c_o :290 */
  o[F_LZ] = (oco_log(ne * (nHI + nHII)) + 2.0 * oco_log(1.0)) - 0.5 * oco_log(t);   /* c_o :292-294 */
  o[F_PAD0] = o[F_PAD1] = 0.0;
}

/* ---- per-wavelength constants ------------------------------------------------------- */
struct Lam {
  double chi, chi1, gff, wa3, s, hmon, f1, f2, f3, gn[6], nu9, l3nu, hnuk, wcm1, sw5;
};

__device__ __forceinline__ void load_lam(Lam &L, const double *__restrict__ lam, int iw, int nw) {
#define LD(f) __ldg(lam + (int64_t)(f) * nw + iw)
  L.chi = LD(L_CHI);
  L.chi1 = LD(L_CHI1);
  L.gff = LD(L_GFF);
  L.wa3 = LD(L_WA3);
  L.s = LD(L_SCOEF);
  L.hmon = LD(L_HMON);
  L.f1 = LD(L_F1);
  L.f2 = LD(L_F2);
  L.f3 = LD(L_F3);
#pragma unroll
  for (int q = 0; q < 6; q++) L.gn[q] = LD(L_GN1 + q);
  L.nu9 = LD(L_NU9);
  L.l3nu = LD(L_L3NU);
  L.hnuk = LD(L_HNUK);
  L.wcm1 = LD(L_WCM1);
  L.sw5 = LD(L_SW5);
#undef LD
}

/* The constants as opacity_at reads them: LamR holds them in registers (loaded from the global
 * table); LamS reads them from the warp's shared-memory table [field][32], one column per lane,
 * which frees ~40 registers of the staged kernel (at 128 no spills but in the ring variants; +3% plain,
 * +5% stable on the AGN grid).  Same values, so the same bits. */
enum { NLF = 20 }; /* fields of the shared table, in the order of store_lam_shared */
struct LamR {
  Lam L;
  template <class IT> __device__ __forceinline__ LamR(const IT &it, const double *, bool load = true) {
    if (load) load_lam(L, it.lam(), it.iw(), it.nw()); /* grey: no wavelength table */
  }
  __device__ __forceinline__ double chi() const { return L.chi; }
  __device__ __forceinline__ double chi1() const { return L.chi1; }
  __device__ __forceinline__ double gff() const { return L.gff; }
  __device__ __forceinline__ double2 wa3_s() const { return make_double2(L.wa3, L.s); }
  __device__ __forceinline__ bool hmon() const { return L.hmon != 0.0; }
  __device__ __forceinline__ double f1() const { return L.f1; }
  __device__ __forceinline__ double f2() const { return L.f2; }
  __device__ __forceinline__ double f3() const { return L.f3; }
  __device__ __forceinline__ double gn(int q) const { return L.gn[q]; }
  __device__ __forceinline__ double nu9() const { return L.nu9; }
  __device__ __forceinline__ double l3nu() const { return L.l3nu; }
  __device__ __forceinline__ double hnuk() const { return L.hnuk; }
  __device__ __forceinline__ double wcm1() const { return L.wcm1; }
  __device__ __forceinline__ double sw5() const { return L.sw5; }
};
struct LamS {
  const double *p; /* &table[0][lane] past the pairs */
  bool hm;
  template <class IT>
  __device__ __forceinline__ LamS(const IT &, const double *table, bool load = true)
      : p(table + 64 + (threadIdx.x & 31)), hm(load && p[3 * 32] != 0.0) {}
  __device__ __forceinline__ double f(int k) const { return p[k * 32]; }
  /* the lane's (wa3, s) pair: two of the constants that every point reads, in one load */
  __device__ __forceinline__ double2 wa3_s() const {
    return *reinterpret_cast<const double2 *>(p - 64 + (threadIdx.x & 31));
  }
  __device__ __forceinline__ double chi() const { return f(0); }
  __device__ __forceinline__ double chi1() const { return f(1); }
  __device__ __forceinline__ double gff() const { return f(2); }
  __device__ __forceinline__ bool hmon() const { return hm; }
  __device__ __forceinline__ double f1() const { return f(4); }
  __device__ __forceinline__ double f2() const { return f(5); }
  __device__ __forceinline__ double f3() const { return f(6); }
  __device__ __forceinline__ double gn(int q) const { return f(7 + q); }
  __device__ __forceinline__ double nu9() const { return f(13); }
  __device__ __forceinline__ double l3nu() const { return f(14); }
  __device__ __forceinline__ double hnuk() const { return f(15); }
  __device__ __forceinline__ double wcm1() const { return f(16); }
  __device__ __forceinline__ double sw5() const { return f(17); }
};
/* Lane's constants in the warp's shared table: the 32 lanes' (wa3, s) pairs, then [field][32]
 * (wavelength iw of the global table). */
__device__ __forceinline__ void store_lam_shared(double *table, int lane, const double *__restrict__ lam, int iw, int nw) {
  const int src[NLF - 2] = {L_CHI, L_CHI1, L_GFF, L_HMON, L_F1, L_F2, L_F3, L_GN1, L_GN2, L_GN3,
                            L_GN4, L_GN5, L_GN6, L_NU9, L_L3NU, L_HNUK, L_WCM1, L_SW5};
  table[2 * lane] = __ldg(lam + (int64_t)L_WA3 * nw + iw);
  table[2 * lane + 1] = __ldg(lam + (int64_t)L_SCOEF * nw + iw);
#pragma unroll
  for (int k = 0; k < NLF - 2; k++) table[64 + k * 32 + lane] = __ldg(lam + (int64_t)src[k] * nw + iw);
}

/* One pillar record, read through the read-only cache (global, 16-byte aligned) or from shared or
 * local memory. */
struct GlobalRec {
  const double *p;
  __device__ __forceinline__ double operator[](int f) const { return __ldg(p + f); }
  __device__ __forceinline__ double2 pair(int f) const { return __ldg(reinterpret_cast<const double2 *>(p + f)); }
};
struct SharedRec {
  const PillarRecord *p;
  __device__ __forceinline__ double operator[](int f) const { return p->f[f]; }
  __device__ __forceinline__ double2 pair(int f) const { return *reinterpret_cast<const double2 *>(p->f + f); }
};

/* Opacity and source function of one (z, lambda), and the absorption fraction w = 1 - albedo
 * (stable form: the ratio of the absorption terms to the sum, no cancellation).  w comes from the
 * quotient num/kr by recip_div.h: where wok is 0 its operands failed the checks and settle_opac
 * divides with the operator.  ook: op lies in the range of the rows' quotients. */
struct Opac {
  double op, w, S;
  double num, kr;
  int wok, ook;
};
template <bool STABLE>
__device__ __forceinline__ void settle_opac(Opac &o) {
  if (!o.wok) {
    const double q = div_call(o.num, o.kr);
    o.w = STABLE ? q : 1.0 - q;
    o.wok = 1;
  }
}
/* Opacities (positive) whose squares, means and ratios stay in the quotients' range. */
__device__ __forceinline__ int op_ok(double op) {
  return ((div_hi(op) - ((uint32_t)(1023 - 159) << 20)) < ((uint32_t)318 << 20)) & div_b_frac_ok(op);
}

/* The factors of a (z, lambda) point that depend on (T, lambda) alone.  A disk's temperature
 * falls to its floor a few scale heights from the midplane (floorTemp of the decks; 85% of the
 * levels of the AGN and Athena-style grids), so the lane keeps the last level's factors and takes
 * them again while the record says that T has not changed by a bit: three exponentials, a
 * division, the level sum and the free-free Gaunt factor less per point, the same bits.
 * AGN grid, 3072 columns x 512 levels x 256 wavelengths, plain: 11.05 -> 7.2 ms; ragged turbulent
 * batch of 400 columns 5.2 -> 3.6 ms; a disk without a floor unchanged (13.7 ms). */
struct TFac {
  double stim, astim, p10f, S, lev, gff; /* astim = AHbf*stim */
};
enum { NTC = 6 };
struct TCacheR { /* in registers (lanes of a warp in different columns) */
  TFac v;
  __device__ __forceinline__ TFac get() const { return v; }
  __device__ __forceinline__ void put(const TFac &t) { v = t; }
};
struct TCacheS { /* the lane's pairs in the warp's shared table [NTC/2][32] */
  double2 *p;
  __device__ __forceinline__ TFac get() const {
    const double2 a = p[0], b = p[32], c = p[64];
    return TFac{a.x, a.y, b.x, b.y, c.x, c.y};
  }
  __device__ __forceinline__ void put(const TFac &t) {
    p[0] = make_double2(t.stim, t.astim);
    p[32] = make_double2(t.p10f, t.S);
    p[64] = make_double2(t.lev, t.gff);
  }
};

/* The rare full evaluations, out of line. */
static __device__ __noinline__ double exp_dd_call(double xh, double xl) { return oco_exp_dd(xh, xl); }
static __device__ __noinline__ double log_call(double x) { return oco_log(x); }

/* calc_opacity_and_albedo for one (z, lambda), continuous_opacity.f90:175-201 with
 * :171, :233-244, :318-322, :337-339, :261-277, :290-298, :399-407. */
/* 10^y1, 10^y2 and e^x3 as oco_pow10, oco_pow10 and oco_exp compute them, with the three
 * fast phases side by side (branch-free, so that their dependency chains overlap) and the
 * full evaluation only where a fast phase cannot decide. */
__device__ __forceinline__ void pow10_pow10_exp(double y1, double y2, double x3, double &r1, double &r2,
                                                double &r3) {
  const double p1 = OCO_M(y1, OCO_LN10_HI), p2 = OCO_M(y2, OCO_LN10_HI);
  const double l1 = OCO_A(OCO_FMA(y1, OCO_LN10_HI, -p1), OCO_M(y1, OCO_LN10_LO));
  const double l2 = OCO_A(OCO_FMA(y2, OCO_LN10_HI, -p2), OCO_M(y2, OCO_LN10_LO));
  double f1, f2, f3;
  const int ok1 = oco_exp_fast_nb(p1, l1, &f1);
  const int ok2 = oco_exp_fast_nb(p2, l2, &f2);
  const int ok3 = oco_exp_fast_nb(x3, 0.0, &f3);
  if (!ok1) f1 = exp_dd_call(p1, l1);
  if (!ok2) f2 = exp_dd_call(p2, l2);
  if (!ok3) f3 = exp_dd_call(x3, 0.0);
  r1 = OCO_M(1.0, f1);
  r2 = OCO_M(1.0, f2);
  r3 = f3;
}

/* bremsstrahlung_absorptionCoeff (c_o :281-300): the Gaunt factor's log, exp and log and the other
 * factor's exp, log and exp side by side without branches (each would be a chain of its own behind
 * its special cases), and the full functions where an argument is not an ordinary one or a fast
 * exponential cannot decide its rounding (a warm disk of 1800 columns x 500 x 250, 62% of the points
 * ionized: 12.6 -> 11.07 ms). */
__device__ __forceinline__ double bremsstrahlung(double a, double b, double c) {
  double a1, b1, a2, b2, a3, b3;
  int ok = oco_log_nb(a, &a1) & oco_exp_fast_nb(b, 0.0, &b1);
  ok &= oco_exp_fast_nb(5.960 - (sqrt3 * pi1) * a1, 0.0, &a2) & oco_log_nb(1.0 - b1, &b2);
  ok &= oco_log_nb(a2 + exp1, &a3) & oco_exp_fast_nb(c + b2, 0.0, &b3);
  if (!ok) {
    a3 = log_call(exp_dd_call(5.960 - (sqrt3 * pi1) * log_call(a), 0.0) + exp1);
    b3 = exp_dd_call(c + log_call(1.0 - exp_dd_call(b, 0.0)), 0.0);
  }
  return (bremsstrahlung_constant * b3) * a3;
}

template <bool STABLE, class R, class LM, class TC>
__device__ __forceinline__ Opac opacity_at(const R P, const LM &L, TC &tc, bool fresh = false) {
  const double2 em = P.pair(F_ESCM);
  const int flags = __double2loint(em.y);
  const bool neutral = flags & FLAG_NEUTRAL;
  TFac t;
  if ((flags & FLAG_SAME_T) && !fresh) { /* fresh: tc does not hold the level below */
    t = tc.get();
  } else {
    double damping = P[F_DFT1] * L.wcm1();
    if (damping > log_overflow_limit) damping = log_overflow_limit;
    double p10_stim, e_planck;
    pow10_pow10_exp(-(L.chi() * P[F_THETA]), ((L.f1() + L.f2() * P[F_LGT]) + L.f3() * P[F_LGT2]) - 26.0, damping,
                    p10_stim, t.p10f, e_planck); /* p10f = 10^(f1 + f2 lgt + f3 lgt^2 - 26) */
    t.stim = 1.0 - p10_stim;
    t.astim = AHbf * t.stim;
    double sm = 0.0;
#pragma unroll
    for (int q = 0; q < 6; q++) sm = sm + L.gn(q) * P[F_E1 + q];
    t.lev = P[F_UNSOLD] + sm;
    t.gff = 1.0 + L.gff() * ((P[F_TH1L] * L.chi1()) + 0.5);
    t.S = L.sw5() / (e_planck - 1.0);
    tc.put(t);
  }
  const double2 ih = P.pair(F_IONF), ae = P.pair(F_AFF), re = P.pair(F_RHO), ws = L.wa3_s();
  const double ionf = ih.x, rho = re.x;
  const double kHbf = ((t.astim * ionf) * ws.x) * t.lev;
  const double kHm = ((ih.y * t.stim) * ionf) * ws.y;
  const double kHmbf = L.hmon() ? kHm : 0.0;
  const double kHmff = ae.x * t.p10f;
  const double abs3 = (kHbf + kHmbf) + kHmff;
  double kr = (abs3 + ae.y) * mp1, op = kr * rho, x;
  if (neutral) {
    x = (((((t.stim * ionf) * alpha0) * ws.x) * t.gff) * re.y) * mp1; /* kHff*mp1 */
    kr = kr + x;
    op = op + kr * rho;
  } else {
    op = op + bremsstrahlung(L.nu9() * P[F_TPOW], -(L.hnuk() * P[F_T1]), P[F_LZ] - L.l3nu());
    x = op * P[F_RHO1];
    kr = kr + x;
  }
  Opac o;
  o.op = op;
  o.kr = kr;
  o.S = t.S;
  o.num = STABLE ? abs3 * mp1 + x : em.x;
  const double q = div_quot(o.num, o.kr, div_recip(o.kr));
  o.w = STABLE ? q : 1.0 - q;
  o.wok = div_b_ok(o.kr) & (STABLE ? div_a_ok(o.num) : (flags & FLAG_ESC_OK) != 0);
  o.ook = op_ok(o.op);
  return o;
}

/* grey_parameters, continuous_opacity.f90:377-390 */
template <bool STABLE, class R>
__device__ __forceinline__ Opac opacity_grey(const R P, double sg) {
  double alpha = P[G_ALPHA];
  Opac o;
  o.op = (alpha + sg) * P[G_RHO];
  o.w = STABLE ? alpha / (alpha + sg) : 1.0 - sg / (alpha + sg);
  o.S = P[G_S];
  o.num = o.kr = 0.0;
  o.wok = 1;
  o.ook = op_ok(o.op);
  return o;
}

/* ---- the solve ----------------------------------------------------------------------- */
/* Issues an L2 prefetch of the line holding p. */
__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p)));
}

/* 1/kappa of a scratch value (see KAPPA_REVERSE), rounded as the division. */
template <class ST>
__device__ __forceinline__ double scratch_o1(double a) {
  if (!ST::KAPPA_REVERSE) return a;
  double y = div_recip(a);
  if (!op_ok(a)) y = div_call(1.0, a);
  return y;
}

/* The sweeps over stored levels load them in two groups of G (4 or 8) that take turns: one is used
 * while the other is in flight.  (A ring whose slots are reloaded one by one waits a full latency
 * per level: a warp has six scoreboards and waits for all loads that share one.)  4 where registers
 * are short and many warps run, 8 where a warp is alone with the latency (k_chain, 16 columns x 500
 * x 250: 455 us with a ring of 8, 281 us with groups of 4, 277 us with 8). */
constexpr int RG = 4, RG_ALONE = 8;

/* U_{k+1} -> U at the level above the returned k, which leaves at least the four bottom levels. */
template <int G>
__device__ __forceinline__ double back_substitute(int &k, double U, const double *__restrict__ gam,
                                                  const double *__restrict__ uu, int64_t ss, int nz) {
  struct Lev {
    double u, g;
  } A[G], B[G];
  auto load = [&](Lev *l, int k0) {
#pragma unroll
    for (int i = 0; i < G; i++) {
      const int kl = max(k0 - i, 0);
      l[i] = Lev{uu[kl * ss], gam[(kl + 1) * ss]};
    }
  };
  auto steps = [&](const Lev *l) {
#pragma unroll
    for (int i = 0; i < G; i++) U = l[i].u - l[i].g * U;
  };
  load(A, k);
#pragma unroll 1
  for (; k >= 2 * G + 3; k -= 2 * G) {
    load(B, k - G);
    steps(A);
    load(A, k - 2 * G);
    steps(B);
  }
  return U;
}

/* The reverse sweep of one item (back-substitution, tridag :43-45; ghost zones :49-62; flux
 * :96-109) from the forward sweep's last u and its scratch (gamma, u, kap: 1/kappa or kappa, and, stable form, q at
 * stride it.ss()), storing U, V (and kappa) through st and the emergent fluxes through the item
 * accessor.  PF: the scratch was written long before (by another kernel) and few warps run, so the
 * next groups are prefetched into L2 as well. */
template <int FORM, int G = RG, bool PF = false, class IT, class ST>
__device__ __forceinline__ void solve_reverse(const IT &it, bool active, double u, const double *__restrict__ gam,
                                              const double *__restrict__ uu, const double *__restrict__ kap,
                                              const double *__restrict__ qs, ST &st) {
  const int nz = it.nz();
  const int64_t ss = it.ss();
  const double dz1 = it.dz1();
  double vtop = 0.0, vbot = 0.0;
  if (FORM == 1 && nz >= 4) {
    /* Stable form: the differences D_k = U_k - U_{k+1} = u_k - q_k U_{k+1} come out of the
     * back-substitution directly, and the flux is the 6th-order stencil written in them
     * (ghost differences mirror the interior ones); exact in the same arithmetic as the
     * stencil on U, accurate where U's differences are below its resolution. */
    const int n = nz;
    st.open(n);
    double Un = u; /* U_{n-1} */
    st.push_u(3, n + 2, Un);
    double Uk[3], Dt[3];
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const int k = n - 2 - t;
      const double uf = uu[k * ss];
      Dt[t] = uf - qs[k * ss] * Un;
      Un = uf - gam[(k + 1) * ss] * Un;
      Uk[t] = Un;
      if (t < 2) st.push_u(4 + t, 3 + k, Un);
    }
    const double fn = u;
    st.push_u(2, n + 3, 2.0 * fn - Uk[0]);
    st.push_u(1, n + 4, 2.0 * fn - Uk[1]);
    st.push_u(0, n + 5, 2.0 * fn - Uk[2]);
    double d0 = Dt[2], d1 = Dt[1], d2 = Dt[0], d3 = Dt[0], d4 = Dt[1], d5 = Dt[2];
    auto flux = [&](double op) -> double {
      const double s1 = d2 + d3;
      const double s2 = (s1 + d1) + d4;
      const double s3 = (s2 + d0) + d5;
      const double df = -((1.0 / 60.0) * (((45.0 * s1) - 9.0 * s2) + s3));
      return ((-1.0 * scratch_o1<ST>(op)) * df) * dz1;
    };
    {
      const double op = kap[(n - 1) * ss];
      vtop = flux(op);
      st.push(6, n - 1, Un, vtop, op); /* U_{n-4}, V_{n-1} */
      st.template group<false>(n - 1, 7);
    }
    double U0 = Uk[2], U1 = Uk[1], U2 = Uk[0], U3 = u; /* the four lowest U seen so far */
    auto step = [&](int slot, int k, double uf, double qk, double gk1, double op) {
      const double Dk = uf - qk * Un;
      Un = uf - gk1 * Un;
      U3 = U2; U2 = U1; U1 = U0; U0 = Un;
      d5 = d4; d4 = d3; d3 = d2; d2 = d1; d1 = d0; d0 = Dk;
      st.push(slot, 3 + k, Un, flux(op), op);
    };
    int k = n - 5;
    struct Lev {
      double u, q, g, o;
    } A[G], B[G];
    auto load = [&](Lev *l, int k0) {
#pragma unroll
      for (int i = 0; i < G; i++) {
        const int kl = max(k0 - i, 0);
        l[i] = Lev{uu[kl * ss], qs[kl * ss], gam[(kl + 1) * ss], kap[(kl + 3) * ss]};
      }
    };
    auto steps = [&](const Lev *l, int slot, int k0) { /* G levels */
#pragma unroll
      for (int i = 0; i < G; i++) step(slot + i, k0 - i, l[i].u, l[i].q, l[i].g, l[i].o);
      if (slot + G == 8) st.template group<true>(3 + k0 - G + 1, 8);
    };
    if (ST::PLANES) /* U alone down to the bottom's last levels */
      Un = back_substitute<G>(k, Un, gam, uu, ss, nz);
    load(A, k);
#pragma unroll 1
    for (; !ST::PLANES && k >= 2 * G - 1; k -= 2 * G) {
      if (PF)
        for (int p = 4 * G; p < 6 * G && k - p >= 0; p++) { /* two pairs of groups ahead into L2 */
          prefetch_l2(&uu[(k - p) * ss]);
          prefetch_l2(&qs[(k - p) * ss]);
          prefetch_l2(&gam[(k - p + 1) * ss]);
          prefetch_l2(&kap[(k - p + 3) * ss]);
        }
      load(B, k - G);
      steps(A, 0, k);
      load(A, k - 2 * G);
      steps(B, G % 8, k - G);
    }
    /* the remaining levels, then the ghosts: 0, 1, 2 levels above the bottom, whose differences
     * D_{-1}, D_{-2}, D_{-3} mirror D_0, D_1, D_2; one level loaded ahead */
    double g0 = 0.0, g1 = 0.0, g2 = 0.0, D1 = 0.0, D2 = 0.0, Dn = 0.0;
    Lev x = A[0];
    int q = 0;
#pragma unroll 1
    for (; k >= -3; k--) {
      if (k >= 0) {
        const int kn = max(k - 1, 0);
        const Lev nx{uu[kn * ss], qs[kn * ss], gam[(kn + 1) * ss], kap[(kn + 3) * ss]};
        step(q, k, x.u, x.q, x.g, x.o);
        x = nx;
      } else {
        if (k == -1) {
          g2 = 2.0 * U0 - U1;
          g1 = 2.0 * U0 - U2;
          g0 = 2.0 * U0 - U3;
          Dn = d0;
          D1 = d1;
          D2 = d2;
        }
        d5 = d4; d4 = d3; d3 = d2; d2 = d1; d1 = d0; d0 = k == -1 ? Dn : (k == -2 ? D1 : D2);
        const double op = kap[(3 + k) * ss];
        vbot = flux(op);
        st.push(q, 3 + k, k == -1 ? g2 : (k == -2 ? g1 : g0), vbot, op);
      }
      if (++q == 8) {
        st.template group<false>(3 + k, 8);
        q = 0;
      }
    }
    st.finish(q);
  } else if (nz >= 4) {
    const int n = nz;
    double u1 = u; /* U_{n-1} */
    double u2 = uu[(n - 2) * ss] - gam[(n - 1) * ss] * u1;
    double u3 = uu[(n - 3) * ss] - gam[(n - 2) * ss] * u2;
    double u4 = uu[(n - 4) * ss] - gam[(n - 3) * ss] * u3;
    double g1 = 2.0 * u1 - u2, g2 = 2.0 * u1 - u3, g3 = 2.0 * u1 - u4;
    st.open(n);
    st.push_u(0, n + 5, g3);
    st.push_u(1, n + 4, g2);
    st.push_u(2, n + 3, g1);
    st.push_u(3, n + 2, u1);
    st.push_u(4, n + 1, u2);
    st.push_u(5, n, u3);
    double w0 = u4, w1 = u3, w2 = u2, w3 = u1, w4 = g1, w5 = g2, w6 = g3;
    auto flux = [&](double op) -> double {
      double df = (1.0 / 60.0) * (((45.0 * (w4 - w2)) - 9.0 * (w5 - w1)) + (w6 - w0));
      return ((-1.0 * scratch_o1<ST>(op)) * df) * dz1;
    };
    {
      const double op = kap[(n - 1) * ss];
      vtop = flux(op);
      st.push(6, n - 1, u4, vtop, op);
      st.template group<false>(n - 1, 7);
    }
    auto step = [&](int slot, int k, double uk, double gk1, double op) {
      double Uk = uk - gk1 * w0;
      w6 = w5; w5 = w4; w4 = w3; w3 = w2; w2 = w1; w1 = w0; w0 = Uk;
      st.push(slot, 3 + k, Uk, flux(op), op);
    };
    int kk = n - 5;
    struct Lev {
      double u, g, o;
    } A[G], B[G];
    auto load = [&](Lev *l, int k0) {
#pragma unroll
      for (int i = 0; i < G; i++) {
        const int kl = max(k0 - i, 0);
        l[i] = Lev{uu[kl * ss], gam[(kl + 1) * ss], kap[(kl + 3) * ss]};
      }
    };
    auto steps = [&](const Lev *l, int slot, int k0) { /* G levels */
#pragma unroll
      for (int i = 0; i < G; i++) step(slot + i, k0 - i, l[i].u, l[i].g, l[i].o);
      if (slot + G == 8) st.template group<true>(3 + k0 - G + 1, 8);
    };
    if (ST::PLANES) w0 = back_substitute<G>(kk, w0, gam, uu, ss, nz);
    load(A, kk);
#pragma unroll 1
    for (; !ST::PLANES && kk >= 2 * G - 1; kk -= 2 * G) {
      load(B, kk - G);
      steps(A, 0, kk);
      load(A, kk - 2 * G);
      steps(B, G % 8, kk - G);
    }
    /* the remaining levels, then the ghosts, one level loaded ahead */
    double b0 = 0.0, b1 = 0.0, b2 = 0.0;
    Lev x = A[0];
    int q = 0;
#pragma unroll 1
    for (; kk >= -3; kk--) {
      if (kk >= 0) {
        const int kn = max(kk - 1, 0);
        const Lev nx{uu[kn * ss], gam[(kn + 1) * ss], kap[(kn + 3) * ss]};
        step(q, kk, x.u, x.g, x.o);
        x = nx;
      } else {
        if (kk == -1) {
          b2 = 2.0 * w0 - w1;
          b1 = 2.0 * w0 - w2;
          b0 = 2.0 * w0 - w3;
        }
        const double b = kk == -1 ? b2 : (kk == -2 ? b1 : b0);
        w6 = w5; w5 = w4; w4 = w3; w3 = w2; w2 = w1; w1 = w0; w0 = b;
        const double op = kap[(3 + kk) * ss];
        vbot = flux(op);
        st.push(q, 3 + kk, b, vbot, op);
      }
      if (++q == 8) {
        st.template group<false>(3 + kk, 8);
        q = 0;
      }
    }
    st.finish(q);
  } else { /* nz = 2 or 3: the reference's ghost update order matters (ghosts feed ghosts) */
    double f[9];
    const int n1 = 3, n2 = nz + 2;
    f[n1 + nz - 1] = u;
    for (int j = nz - 2; j >= 0; j--) f[n1 + j] = uu[j * ss] - gam[(j + 1) * ss] * f[n1 + j + 1];
    for (int i = 1; i <= 3; i++) {
      f[n1 - i] = 2.0 * f[n1] - f[n1 + i];
      f[n2 + i] = 2.0 * f[n2] - f[n2 - i];
    }
    for (int m = 0; m < nz + 6; m++) st.u(m, f[m]);
    for (int j = 0; j < nz; j++) {
      int c = n1 + j;
      double df = (1.0 / 60.0) * (((45.0 * (f[c + 1] - f[c - 1])) - 9.0 * (f[c + 2] - f[c - 2])) +
                                  (f[c + 3] - f[c - 3]));
      const double op = kap[j * ss];
      double v = ((-1.0 * scratch_o1<ST>(op)) * df) * dz1;
      st.v(j, v);
      if (ST::KAPPA_REVERSE) st.k(j, op);
      if (j == 0) vbot = v;
      if (j == nz - 1) vtop = v;
    }
  }
  if (!active) return;
  if (double *p = it.vtop()) __stcs(p, vtop);
  if (double *p = it.vbot()) __stcs(p, vbot);
}

/* State of the forward elimination between two rows, and the operand checks of the quotients that
 * the next row forms with it (recip_div.h). */
struct Elim {
  double c;      /* c of the row */
  double h;      /* stable form: h of the row */
  double d;      /* divisor of the next row's quotients: bet (plain) or c + h = -bet (stable) */
  double u;      /* u of the row */
  double kh;     /* mean opacity between the row and the next */
  double yd, yk; /* 1/d, 1/kh */
  int ok;        /* d, c, (h) and kh pass the checks */
};
/* What a row leaves in the scratch beside u: gamma, (stable) q of the row below, 1/kappa. */
struct RowOut {
  double g, q, o1;
};

/* ook: the opacities on both sides of kh pass op_ok. */
template <int FORM>
__device__ __forceinline__ void elim_checks(Elim &e, int ook) {
  e.yd = div_recip(e.d);
  e.yk = div_recip(e.kh);
  e.ok = ook & div_b_ok(e.d) & div_a_ok(e.c) & div_b_frac_ok(e.kh);
  if (FORM == 1) e.ok &= div_a_ok(e.h);
}

/* Centre row (fill_center_coeffs :159-165; tridag :34-40 or its difference form
 * bet = -(c + h), h = e + a h_prev/(c_prev + h_prev)) from the row below's state, with every
 * quotient from a shared reciprocal: c and a share the mean opacities' reciprocals with the
 * neighbouring rows; gamma and u the pivot's (plain); gamma, q, a h and u the same divisor's
 * (stable; -bet of a row is the next row's c + h).  Returns whether every operand passed its
 * check (kh lies between two opacities that did; c, an opacity squared over a mean, is then in
 * range). */
template <int FORM>
__device__ __forceinline__ int center_fast(const Elim &e, const Opac &cur, const Opac &nxt, double dz2, Elim &n,
                                           RowOut &r) {
  const double op = cur.op, o2 = op * op;
  r.o1 = div_recip(op); /* dead where the scratch holds kappa */
  n.kh = 0.5 * (nxt.op + op);
  n.yk = div_recip(n.kh);
  const double aa = div_quot(o2, e.kh, e.yk), cc = div_quot(o2, n.kh, n.yk);
  const double z3 = (dz2 * (op * (op * op))) * cur.w;
  const double dd = -(cur.S * z3);
  const double num = dd - aa * e.u;
  int ok = e.ok & div_a_ok(num);
  n.c = cc;
  if (FORM == 0) {
    const double bb = -((aa + cc) + z3);
    r.g = div_quot(e.c, e.d, e.yd);
    r.q = 0.0;
    n.h = 0.0;
    n.d = bb - aa * r.g;
    n.yd = div_recip(n.d);
    n.u = div_quot(num, n.d, n.yd);
    n.ok = div_b_ok(n.d);
  } else {
    const double ah = aa * e.h;
    r.g = -div_quot(e.c, e.d, e.yd);
    r.q = div_quot(e.h, e.d, e.yd);
    n.h = z3 + div_quot(ah, e.d, e.yd);
    n.d = cc + n.h;
    n.yd = div_recip(n.d);
    n.u = -div_quot(num, n.d, n.yd);
    n.ok = div_b_ok(n.d) & div_a_ok(n.h);
    ok &= div_a_ok(ah);
  }
  n.ok &= nxt.ook & div_b_frac_ok(n.kh);
  return ok & n.ok;
}

/* The same row with the division operator. */
template <int FORM>
__device__ __forceinline__ void center_slow(const Elim &e, const Opac &cur, const Opac &nxt, double dz2, Elim &n,
                                            RowOut &r, bool &bad) {
  const double op = cur.op, o2 = op * op;
  r.o1 = div_call(1.0, op);
  n.kh = 0.5 * (nxt.op + op);
  const double aa = div_call(o2, e.kh), cc = div_call(o2, n.kh);
  const double z3 = (dz2 * (op * (op * op))) * cur.w;
  const double dd = -(cur.S * z3);
  n.c = cc;
  double bet;
  if (FORM == 0) {
    const double bb = -((aa + cc) + z3);
    r.g = div_call(e.c, e.d);
    r.q = 0.0;
    n.h = 0.0;
    n.d = bet = bb - aa * r.g;
  } else {
    r.g = -div_call(e.c, e.d);
    r.q = div_call(e.h, e.d);
    n.h = z3 + div_call(aa * e.h, e.d);
    n.d = cc + n.h;
    bet = -n.d;
  }
  if (bet == 0.0) bad = true;
  n.u = div_call(dd - aa * e.u, bet);
  elim_checks<FORM>(n, cur.ook & nxt.ook);
}

/* The elimination over rows whose coefficients are given (the split block solve and the mixed form's
 * re-solve): state between two rows, d as in Elim. */
struct Chain {
  double c, h, d, yd, u;
  int ok; /* c, (h) and d pass the checks */
};
template <int FORM>
__device__ __forceinline__ void chain_checks(Chain &e) {
  e.yd = div_recip(e.d);
  e.ok = div_b_ok(e.d) & div_a_ok(e.c);
  if (FORM == 1) e.ok &= div_a_ok(e.h);
}
/* Row 0: x is its diagonal (plain) or h (stable). */
template <int FORM>
__device__ __forceinline__ Chain chain_first(double x, double cc, double dd, bool &bad) {
  Chain e;
  e.c = cc;
  e.h = FORM == 0 ? 0.0 : x;
  e.d = FORM == 0 ? x : cc + x;
  const double bet = FORM == 0 ? x : -e.d;
  if (bet == 0.0) bad = true;
  e.u = dd / bet;
  chain_checks<FORM>(e);
  return e;
}
/* A row above: x is its diagonal (plain) or its diagonal excess (stable).  The serial chain is one
 * reciprocal, one quotient and two operations per row (plain; stable: one more quotient's), where
 * the operator's divisions put 2 x 124 cycles and their branches on it. */
template <int FORM>
__device__ __forceinline__ void chain_step(Chain &e, double aa, double x, double cc, double dd, double &g, double &q,
                                           bool &bad) {
  Chain n;
  const double num = dd - aa * e.u;
  int ok = e.ok & div_a_ok(num);
  n.c = cc;
  if (FORM == 0) {
    g = div_quot(e.c, e.d, e.yd);
    q = n.h = 0.0;
    n.d = x - aa * g;
    n.yd = div_recip(n.d);
    n.u = div_quot(num, n.d, n.yd);
  } else {
    const double ah = aa * e.h;
    g = -div_quot(e.c, e.d, e.yd);
    q = div_quot(e.h, e.d, e.yd);
    n.h = x + div_quot(ah, e.d, e.yd);
    n.d = cc + n.h;
    n.yd = div_recip(n.d);
    n.u = -div_quot(num, n.d, n.yd);
    ok &= div_a_ok(ah);
  }
  const int dok = div_b_ok(n.d);
  n.ok = dok & div_a_ok(cc);
  if (FORM == 1) n.ok &= div_a_ok(n.h);
  if (!(ok & dok)) { /* as above with the operator */
    double bet;
    if (FORM == 0) {
      g = div_call(e.c, e.d);
      n.d = bet = x - aa * g;
    } else {
      g = -div_call(e.c, e.d);
      q = div_call(e.h, e.d);
      n.h = x + div_call(aa * e.h, e.d);
      n.d = cc + n.h;
      bet = -n.d;
    }
    if (bet == 0.0) bad = true;
    n.u = div_call(num, bet);
    chain_checks<FORM>(n);
  }
  e = n;
}

/* Levels are bound by dependent FP64 latency, not by a pipe: a warp alone on its SM needed as long
 * per level (~3900 cycles) as sixteen.  So the sweep keeps its chains short and side by side:
 * factors of an unchanged temperature are kept (TFac), a row's seven (plain) or ten (stable)
 * quotients come from four reciprocals without branches, with one check per row
 * (without the kept factors: AGN grid plain 11.84 -> 11.05 ms, 16 columns x 500 x 250 stable
 * 1.03 -> 0.80 ms; with them 7.2 and 0.49 ms).  The GPU then runs this kernel at its 1000 W limit
 * (1.82 GHz), so what counts is instructions per point: records, kept factors and constants are
 * read in 16-byte pairs and the record pointer is advanced instead of computed: 7.48 -> 7.37 ms,
 * 0.49 -> 0.41 ms, batch of 400 columns 3.67 -> 3.53 ms.  Not faster: row j's elimination beside the opacity of level j + 2
 * (7.53 ms; 0.39 ms), the exponentials and logarithms behind calls (7.45; 14.5 for 13.6 ms on the
 * warm disk), five blocks per SM at 96 registers (7.8 ms). */
template <int FORM, bool GREY, class IT, class PA, class LMT, class TC, class ST>
__device__ __forceinline__ void solve_item(const IT &it, bool active, PA &pa, double *__restrict__ gam,
                                           double *__restrict__ uu, double *__restrict__ kap,
                                           double *__restrict__ qs, const double *lam_table, TC tc, ST st) {
  const int nz = it.nz();
  const int64_t ss = it.ss();
  const LMT L(it, lam_table, !GREY);
  const double dz = it.dz(), dz2 = it.dz2();
  bool bad = false;
  auto opac = [&](int z) -> Opac {
    if (GREY) return opacity_grey<FORM == 1>(pa.at(z), it.sigma_grey());
    return opacity_at<FORM == 1>(pa.at(z), L, tc);
  };

  /* forward sweep: row 0 (fill_boundary_coeffs :187-191) */
  Opac cur = opac(0), nxt = opac(1);
  settle_opac<FORM == 1>(cur);
  settle_opac<FORM == 1>(nxt);
  Elim e;
  {
    const double o1 = 1.0 / cur.op, o2 = cur.op * cur.op;
    const double zeta = ((cur.op * dz2) * cur.w) * 0.25;
    double bet;
    e.c = cur.op;
    if (FORM == 0) {
      e.h = 0.0;
      e.d = bet = -(((o1 + dz) + zeta) * o2);
    } else {
      e.h = (dz + zeta) * o2;
      e.d = cur.op + e.h;
      bet = -e.d;
    }
    if (bet == 0.0) bad = true;
    e.u = (-((cur.S * zeta) * o2)) / bet;
    e.kh = 0.5 * (nxt.op + cur.op); /* kappa_p(1) = kappa_m(2), :147-154 */
    elim_checks<FORM>(e, cur.ook & nxt.ook);
    uu[0] = e.u;
    kap[0] = ST::KAPPA_REVERSE ? cur.op : o1;
    if (!ST::KAPPA_REVERSE) st.k(0, cur.op);
  }
  auto put = [&](int j, const RowOut &r, double u, double op) {
    gam[j * ss] = r.g;
    uu[j * ss] = u;
    if (!ST::PLANES || j == nz - 1) kap[j * ss] = ST::KAPPA_REVERSE ? op : r.o1;
    if (!ST::KAPPA_REVERSE) st.k(j, op);
    if (FORM == 1) qs[(j - 1) * ss] = r.q;
  };
  for (int j = 1; j < nz - 1; j++) {
    cur = nxt;
    nxt = opac(j + 1);
    Elim n;
    RowOut r;
    if (!(center_fast<FORM>(e, cur, nxt, dz2, n, r) & nxt.wok)) {
      settle_opac<FORM == 1>(nxt);
      center_slow<FORM>(e, cur, nxt, dz2, n, r, bad);
    }
    put(j, r, n.u, cur.op);
    e = n;
  }
  { /* fill_boundary_coeffs :193-197 */
    const double op = nxt.op, o2 = op * op;
    const double zt = ((op * dz2) * nxt.w) * 0.25;
    const double dd = -((nxt.S * zt) * o2);
    RowOut r;
    double bet;
    r.o1 = 1.0 / op;
    if (FORM == 0) {
      r.g = e.c / e.d;
      r.q = 0.0;
      bet = -(((r.o1 + dz) + zt) * o2) - op * r.g;
    } else {
      r.g = -(e.c / e.d);
      r.q = e.h / e.d; /* q_{j-1} = h_{j-1}/(c_{j-1} + h_{j-1}) */
      bet = -(0.0 + ((dz + zt) * o2 + (op * e.h) / e.d));
    }
    if (bet == 0.0) bad = true;
    e.u = (dd - op * e.u) / bet;
    put(nz - 1, r, e.u, op);
  }
  if (active && bad) {
    atomicAdd(&it.status()[0], 1ull);
    atomicMin(&it.status()[1], it.id());
  }
  __syncwarp();
  solve_reverse<FORM>(it, active, e.u, gam, uu, kap, qs, st);
}

}  // namespace oco

#endif
