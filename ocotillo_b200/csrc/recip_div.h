/*
 * recip_div.h -- correctly rounded FP64 quotients from a shared reciprocal, without branches.
 *
 * The elimination divides several numerators by one divisor (gamma_{j+1} and u_j by the pivot,
 * c_j and a_{j+1} by the mean opacity, the stable form's gamma, q, a h and u by one
 * denominator).  The compiler's division costs a warp ~124 cycles on sm_100a whether or not
 * anything waits for it (its branch for special operands keeps independent divisions from
 * overlapping), so a level with seven of them spends most of its ~4000 cycles there.  Here the
 * divisor's correctly rounded reciprocal is computed once (a seed and five FMAs) and each
 * quotient takes three operations, all in one basic block.
 *
 * Method (P. Markstein, IBM J. Res. Dev. 34(1) 1990; M. Cornea-Hasegan, R. Golliver and
 * P. Markstein, ARITH 1999; Muller et al., Handbook of Floating-Point Arithmetic, 2nd ed.,
 * section 4.7): with 1 <= b < 2 (scaling by powers of two changes nothing in range),
 *   y1 = y0 (1 + e + e^2), e = 1 - b y0, is within 0.6 ulp of 1/b for a seed of relative error
 *        below 2^-19 (e^3 < 2^-57);
 *   y  = RN(y1 + (1 - b y1) y1) is RN(1/b): the computed sum misses 1/b by b t^2 2^-53 ulp, t
 *        the error of y1 in ulps, and at a rounding boundary (t = 1/2) that is b 2^-55 ulp,
 *        while 1/b stays 2^-53/b ulp away from it; b^2 < 4 makes the first smaller;
 *   q0 = RN(a y) is within a/2 + 1/2 ulp of a/b if a < b and within a/4 + 1/2 ulp if a >= b;
 *   q  = RN(q0 + r y), r = a - b q0, is RN(a/b): at the rounding boundary half an ulp from q0
 *        r is exact and y's relative error (at most b 2^-54) moves the sum by b 2^-55 ulp,
 *        while a/b stays 2^-53/b ulp away.  The next boundary, 3/2 ulp away, is out of reach
 *        unless a < b with both within 2^-20 of 2: divisors whose 20 leading fraction bits are
 *        all ones are left to the division operator (div_b_ok).
 * The exponent checks keep every intermediate normal and r exact.  Where a check fails (zero,
 * subnormal, infinite and NaN operands among them) the caller divides with the operator, so
 * every quotient is the IEEE one.
 */
#ifndef OCO_RECIP_DIV_H
#define OCO_RECIP_DIV_H

#include "ocomath.h"

/* Reciprocal seed of relative error below 2^-19: the hardware's approximation (its 20 leading
 * bits), or on the host 1/b cut to as many. */
OCO_HD double div_seed(double b) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
#else
  return oco_u2d(oco_d2u(1.0 / b) & 0xffffffff00000000ULL);
#endif
}

/* RN(1/b) for a divisor that passes div_b_ok. */
OCO_HD double div_recip(double b) {
  const double y0 = div_seed(b);
  const double e = OCO_FMA(-b, y0, 1.0);
  const double y1 = OCO_FMA(y0, OCO_FMA(e, e, e), y0);
  return OCO_FMA(y1, OCO_FMA(-b, y1, 1.0), y1);
}

/* RN(a/b) from y = div_recip(b), for operands that pass the checks below. */
OCO_HD double div_quot(double a, double b, double y) {
  const double q0 = OCO_M(a, y);
  return OCO_FMA(OCO_FMA(-b, q0, a), y, q0);
}

OCO_HD uint32_t div_hi(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2hiint(x);
#else
  return (uint32_t)(oco_d2u(x) >> 32);
#endif
}

/* Whether 2^-lo <= |x| < 2^hi (one shift-add and one unsigned comparison on the high word). */
OCO_HD int div_in_range(double x, int lo, int hi) {
  return ((div_hi(x) << 1) - ((uint32_t)(1023 - lo) << 21)) < ((uint32_t)(lo + hi) << 21);
}

/* Whether b's 20 leading fraction bits are not all ones. */
OCO_HD int div_b_frac_ok(double b) { return ((div_hi(b) + 1u) & 0xfffffu) != 0u; }

/* Divisor check: with |b| in [2^-200, 2^200) and numerators in [2^-760, 2^480) the quotient's
 * magnitude lies in [2^-961, 2^681), and r, whose last bit is at or above 2^-105 of the
 * numerator's leading one, is exact. */
OCO_HD int div_b_ok(double b) { return div_in_range(b, 200, 200) & div_b_frac_ok(b); }
OCO_HD int div_a_ok(double a) { return div_in_range(a, 760, 480); }

#ifdef __CUDACC__
/* The operator where a check fails, out of line: the fast paths around it stay small enough for the
 * instruction caches. */
static __device__ __noinline__ double div_call(double a, double b) { return a / b; }
#endif

#endif /* OCO_RECIP_DIV_H */
