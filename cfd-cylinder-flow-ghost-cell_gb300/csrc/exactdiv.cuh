// a / b in double precision for a divisor known in advance.
#pragma once
#include <cmath>

namespace gmk {

// 1 / b for div_by; NaN for a divisor that is not positive or near the ends of the exponent range (div_by then divides)
inline double reciprocal_of(double b) { return b > 1e-100 && b < 1e100 ? 1.0 / b : std::nan(""); }

// The correctly rounded quotient from rb = reciprocal_of(b): one multiplication and two fused
// multiply-adds (Brisebarre, Muller and Raina, "Accelerating correctly rounded floating-point division
// when the divisor is known in advance", IEEE Trans. Computers 53, 2004), a third of a divide's FP64
// instructions on a device that issues FP64 at 1/64 of the FP32 rate.  The remainder has to be exact, so
// operands and quotients near the ends of the exponent range (and infinities, NaN) take the divide;
// zeros keep their sign.
__device__ __forceinline__ bool div_by_range(double v) {
  return (((unsigned)__double2hiint(v) >> 20) & 0x7ffu) - 128u <= 2046u - 256u;
}
// (a call, so that the compiler does not work out the divide beside the quotients that need none)
static __device__ __noinline__ double div_by_rest(double a, double b, double q) {
  const unsigned hi = (unsigned)__double2hiint(a), qhi = (unsigned)__double2hiint(q);
  const bool zero = ((hi << 1) | (unsigned)__double2loint(a)) == 0 && ((qhi << 1) | (unsigned)__double2loint(q)) == 0;
  return zero ? q : a / b;
}
__device__ __forceinline__ double div_by(double a, double b, double rb) {
  const double q = __dmul_rn(a, rb);
  if (div_by_range(a) && div_by_range(q)) return __fma_rn(__fma_rn(-q, b, a), rb, q);
  return div_by_rest(a, b, q);
}

}  // namespace gmk
