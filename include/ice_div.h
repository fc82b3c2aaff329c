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
 * Why it is the IEEE quotient: let m in [1, 2) be the significand of b. recip's last step leaves y within
 * (1/2 + 2^-24) ulp of 1/b, a relative error of 2^-54 m. quot's first correction leaves q within
 * (1/2 + 2^-50) ulp of a/b; its remainder a - b q is exact. The last step rounds q + r y, which is a/b
 * moved by at most 2^-55 m ulp, while a/b is at least 2^-53 / m ulp from any midpoint of two doubles: the
 * move is the smaller for every m but those next to 2, of which only the largest, all ones, is rounded
 * wrongly (for powers of two above it). ice_div_by excludes it. tests/test_div.py checks the rest against
 * `/`, significands next to 1 and 2 included.
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

/* x is a divisor of the quotients below: the same range, and its low word is not all ones. */
ICE_DIV_FN int ice_div_by(double x) {
#ifdef __CUDA_ARCH__
  const unsigned lo = (unsigned)__double2loint(x);
#else
  union { double d; unsigned long long u; } v;
  v.d = x;
  const unsigned lo = (unsigned)v.u;
#endif
  return ice_div_in(x) && lo != 0xffffffffu;
}

/* The first approximation of 1/b, good to 2^-20 or better (rcp.approx.ftz.f64 on the device). */
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
