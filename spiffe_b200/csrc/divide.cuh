// spiffe_b200/csrc/divide.cuh -- FP64 quotients by a number known beforehand.
#pragma once

// x / e, correctly rounded, for e whose correctly rounded reciprocal is y:
// Markstein's theorem (IBM J. Res. Dev. 34, 1990): a quotient within one unit
// in the last place plus its exactly formed remainder times y rounds to the
// quotient; the first correction brings x*y within that unit.
__device__ __forceinline__ double div_const(double x, double e, double y)
{
  double q = x * y;
  q = __fma_rn(__fma_rn(-q, e, x), y, q);
  return __fma_rn(__fma_rn(-q, e, x), y, q);
}

// Whether x lies outside the range in which div_const's remainders are exact
// (below 2^-940 or above 2^900; x = 0 is inside), by its exponent.
__device__ __forceinline__ bool div_rare(double x)
{
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
  return h - (83u << 20) >= (1840u << 20) && (h | (unsigned)__double2loint(x)) != 0;
}

// x / e there: a tiny x is scaled by a power of two first; that rounds a
// subnormal quotient a second time, which can only matter where the scaled
// one lies half way between two of them.  There, and for infinities and NaN,
// the division.
static __device__ __noinline__ double div_scaled(double x, double e, double y)
{
  const double w = div_const(x * 0x1p500, e, y), q = w * 0x1p-500;
  return !(fabs(x) < 0x1p-900) || fabs(w - q * 0x1p500) == 0x1p-575 ? x / e : q;
}

// x / e with x's sign at x = 0, for 2^-60 <= e <= 2^60 and its reciprocal y
__device__ __forceinline__ double div_by(double x, double e, double y)
{
  if (div_rare(x))
    return div_scaled(x, e, y);
  const double q = div_const(x, e, y);
  return x == 0 ? x : q;
}
inline bool div_by_takes(double e) { return e >= 0x1p-60 && e <= 0x1p60; }
