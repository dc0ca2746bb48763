// mh_div.h -- correctly rounded single-precision quotients by a divisor whose
// reciprocal is known.
//
// P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34 (1990): with y = RN(1 / b) and
// q within one unit in the last place of a / b, RN(q + RN(a - b q) y) is
// RN(a / b), the residual being exact in a fused multiply-add.  RN(a y) may be
// off by one and a half units, so one such step makes it good enough and a
// second one rounds it.  Nothing may over- or underflow (mh_div_ok).  Five
// instructions, where the general division takes about twice that and a branch.
#pragma once
#include <cmath>

#if defined(__CUDACC__)
#define MH_DIV_HD __host__ __device__ __forceinline__
#else
#define MH_DIV_HD static inline
#endif

// a / b for y = 1 / b rounded to nearest
MH_DIV_HD float mh_div(float a, float b, float y) {
  float q = a * y;
  q = fmaf(fmaf(-b, q, a), y, q);
  return fmaf(fmaf(-b, q, a), y, q);
}
// Whether mh_div is exact for these dividends and a divisor within
// 2^-60 .. 2^60, which every length in metres is: quotients stay within
// 2^-120 .. 2^120, and the residuals are multiples of 2^-48 of the dividend, so
// of 2^-108.  (A zero takes the other way, which is right for it too.)
MH_DIV_HD bool mh_div_ok(float a, float b, float c) {
  const float x = fabsf(a), y = fabsf(b), z = fabsf(c);
  return fminf(fminf(x, y), z) > 1e-18f && fmaxf(fmaxf(x, y), z) < 1e18f;
}
