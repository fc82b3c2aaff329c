/* ice_div.h -- correctly rounded FP64 quotients without a branch, so that the quotients of a cell's
 * variables can be evaluated side by side.
 *
 * A compiled FP64 division tests its operands and branches to a general path; a sequence of them runs one
 * after the other, each a chain of dependent operations. Here the quotient is formed by Newton steps on an
 * approximate reciprocal and two corrections with exact remainders (P. Markstein, "Computation of elementary
 * functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990; J.-M. Muller et al.,
 * "Handbook of Floating-Point Arithmetic", the chapter on division by an FMA), for operands whose exponents
 * keep every intermediate value normal. ice_div_in and ice_div_by say whether they do; the caller
 * divides with `/` otherwise. The result is then the IEEE quotient, bit for bit (a zero dividend gives +0 or -0).
 *
 * Why it is the IEEE quotient: let m = 2 - j 2^-52 in [1, 2) be the significand of b and e0 the relative error of the
 * first approximation: on one B200 2^-19.93 at most over every upper word, 2^-21 where the upper twenty bits of the
 * significand are ones (j <= 2^32). Two Newton steps leave e0^4, below 2^-79.6 and for j <= 2^32 below 2^-79.9 (from
 * 2^-20 on), and the last rounding: y = (1 + t) / b, |t| <= 2^-54 m + e0^4, half an ulp of 1/b (whose significand is 2 / m)
 * and the rest.
 * quot's first correction leaves q within (1/2 + 2^-50) ulp of a/b, so its remainder a - b q is exact. The last step
 * rounds q + r y: a/b moved by at most (1/2 + 2^-50) |t| ulp. A quotient of two doubles is at least 2^-53 / m ulp
 * from any midpoint, which leaves 2^-55 (4 - m^2) / m >= j 2^-106 ulp for t beyond 2^-54 m and for the 2^-50.
 *   j > 2^32: 2^-74 and more is left, 2^-80.6 + 2^-103 taken.
 *   2^26 < j <= 2^32: 2^-80 and more is left, 2^-80.9 + 2^-103 taken.
 *   2^14 < j <= 2^26: 1/b has the significand 1 + j h + j^2 h^2 + ..., h = 2^-53, ulp 2 h: for odd j it lies j^2 h^2 > 2^-78
 *     above a tie of doubles, for even j more than 2^-55 off one, so y is 1/b rounded correctly and t has no rest; 2^-92 and
 *     more is left, 2^-103 taken.
 *   j <= 2^14: y may fall on the other side of its tie, and some quotients next to a midpoint are then rounded
 *     wrongly. ice_div_by excludes them by the low word, of every divisor.
 * tests/test_div.py and tests/test_div_midpoints.py check it against `/`.
 */
#ifndef ICE_DIV_H
#define ICE_DIV_H

#ifdef __CUDACC__
#define ICE_DIV_FN __host__ __device__ __forceinline__
#else
#include <math.h>
#define ICE_DIV_FN static inline
#endif

/* The high word of x without its sign: biased exponent in bits 20..30. */
ICE_DIV_FN unsigned ice_div_hi(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(x) & 0x7fffffffu;
#else
  union { double d; unsigned long long u; } v;
  v.d = x;
  return (unsigned)(v.u >> 32) & 0x7fffffffu;
#endif
}

/* 2^-200 <= |x| < 2^200: x is a dividend of the quotients below (and zero is one). */
ICE_DIV_FN int ice_div_in(double x) { return ice_div_hi(x) - (823u << 20) < (400u << 20); }

/* The low words of the divisors with j <= 2^14. */
#define ICE_DIV_LOW 0xffffc000u

ICE_DIV_FN unsigned ice_div_lo(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(x);
#else
  union { double d; unsigned long long u; } v;
  v.d = x;
  return (unsigned)v.u;
#endif
}

/* j <= 2^14 */
ICE_DIV_FN int ice_div_top(double x) { return ice_div_lo(x) >= ICE_DIV_LOW && (~ice_div_hi(x) & 0xfffffu) == 0u; }

/* x is a divisor of the quotients below: the same range, and by its low word not one with j <= 2^14. */
ICE_DIV_FN int ice_div_by(double x) { return ice_div_in(x) && ice_div_lo(x) < ICE_DIV_LOW; }

/* The first approximation of 1/b (rcp.approx.ftz.f64 on the device; its error: see above). */
ICE_DIV_FN double ice_div_seed(double b) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
#else
  return (double)(1.0f / (float)(b));    /* the host's check only: |b| within a float's range */
#endif
}

ICE_DIV_FN double ice_div_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return fma(a, b, c);
#endif
}

/* 1/b from a first approximation y. */
ICE_DIV_FN double ice_div_refine(double b, double y) {
  double e = ice_div_fma(-b, y, 1.0);
  y = ice_div_fma(e, y, y);
  e = ice_div_fma(-b, y, 1.0);
  return ice_div_fma(e, y, y);
}

ICE_DIV_FN double ice_div_recip(double b) { return ice_div_refine(b, ice_div_seed(b)); }

/* a / b from y = ice_div_recip(b). */
ICE_DIV_FN double ice_div_quot(double a, double b, double y) {
#ifdef __CUDA_ARCH__
  double q = __dmul_rn(a, y);
#else
  double q = a * y;
#endif
  double r = ice_div_fma(-b, q, a);
  q = ice_div_fma(r, y, q);
  r = ice_div_fma(-b, q, a);
  return ice_div_fma(r, y, q);
}

#endif
