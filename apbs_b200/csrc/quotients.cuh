// Quotients and reciprocals by multiplication, for kernels whose step waits for one.
#pragma once
#include "common.cuh"

namespace pmgb {

// The factor div_by takes for divisor b: RN(1 / b), or NaN (div_by then divides)
// where b is so large or small that a remainder could underflow or overflow.
__device__ __forceinline__ double div_factor(double b) {
  const double m = fabs(b);
  return m >= 0x1p-200 && m <= 0x1p200 ? 1.0 / b : __longlong_as_double(0x7ff8000000000000ll);
}

// a / b, correctly rounded, with y = div_factor(b): P. Markstein's quotient (IBM J.
// Res. Dev. 34, 1990): with y correctly rounded, a quotient within one ulp of a / b
// is corrected to the rounded one by its exact remainder times y; the first
// correction brings a*y (up to 1.5 ulp off) there.  Outside the quotients of 2^-767
// to 2^769, and where y is NaN, the division itself.  Equal to a / b bit for bit
// (tests/test_gpu_quotients.py).
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q0 = a * y;
  const double q1 = __fma_rn(__fma_rn(-b, q0, a), y, q0);
  const double q2 = __fma_rn(__fma_rn(-b, q1, a), y, q1);
  const unsigned e = (unsigned)__double2hiint(q0) & 0x7fffffffu;  // exponent of the quotient
  if (e - 0x10000000u < 0x60000000u) return q2;
  if (a == 0.0 && q0 == 0.0) return q0;  // 0 / b, of either sign
  return a / b;
}

// 1 / x to an ulp for normal x of 2^-1000 to 2^1000, by Newton's iteration on the
// hardware's approximation (20 bits): two steps reach 80 bits in exact arithmetic,
// the third takes out the rounding of the second.
__device__ __forceinline__ double reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(fma(-x, y, 1.0), y, y);
  y = fma(fma(-x, y, 1.0), y, y);
  return fma(fma(-x, y, 1.0), y, y);
}

}  // namespace pmgb
