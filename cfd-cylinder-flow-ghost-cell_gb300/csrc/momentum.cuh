// The AB2 momentum right-hand side at a face away from the channel's edges (FP64).
#pragma once
#include <cmath>

namespace gmk {

// What multiplies the unscaled products, formed on the host.
struct MomentumC {
  double ax, ay;       // -dy / (4 dx dy), -dx / (4 dx dy): of the products' differences along x and y
  double c1, c2;       // dt (1 + alpha), dt alpha
  double lx, ly;       // dt nu / (2 dx^2), dt nu / (2 dy^2)
  double gx, gy;       // dt / (rho dx), dt / (rho dy)
};

// x plus the step's increment, from the neighbours' sums ew and ns, the advection now and before and the
// pressure's part dp.  The increment is formed by itself and added last, so it alone is rounded against x: a
// constant field stays as it is to the bit.  (With x in the products, as lc x + lx ew + ly ns, two
// instructions of fifteen are saved, but lc's rounding moves the field by up to an ulp a step, always
// to the same side.)
__host__ __device__ __forceinline__ double momentum_rhs(const MomentumC& m, double x, double ew, double ns, double now, double prev,
                                                       double dp) {
  return x + fma(m.lx, fma(-2.0, x, ew), fma(m.ly, fma(-2.0, x, ns), fma(m.c1, now, fma(-m.c2, prev, -dp))));
}

}  // namespace gmk
