// Host check of momentum.cuh: a constant field without advection or pressure gradient stays as it is to the
// bit, and the right-hand side is within half an ulp of its own and the increment's roundings of the exact value.
// Built and run by tests/test_momentum_rhs.py.
#include <cstdio>
#include <random>

#include "momentum.cuh"
using namespace gmk;
int main() {
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0), e(-3.0, 0.0);
  long moved = 0, far = 0;
  for (int k = 0; k < 200000; ++k) {
    const double dt = std::pow(10.0, e(rng) - 1), nu = std::pow(10.0, e(rng)), dx = std::pow(10.0, e(rng) / 2 - 0.5);
    const double dy = dx * (1.5 + u(rng)), alpha = 0.5 + 0.4 * u(rng);
    MomentumC m{};
    m.c1 = dt * (1 + alpha);
    m.c2 = dt * alpha;
    m.lx = 0.5 * dt * nu / (dx * dx);
    m.ly = 0.5 * dt * nu / (dy * dy);
    const double c = u(rng);
    if (momentum_rhs(m, c, c + c, c + c, 0.0, 0.0, 0.0) != c) ++moved;
    const double ew = 2 * u(rng), ns = 2 * u(rng), now = u(rng), prev = u(rng), dp = 0.1 * u(rng);
    const long double a = (long double)m.lx * ((long double)ew - 2.0L * c), b = (long double)m.ly * ((long double)ns - 2.0L * c);
    const long double p = (long double)m.c1 * now, q = (long double)m.c2 * prev;
    const long double inc = a + b + p - q - dp, size = fabsl(a) + fabsl(b) + fabsl(p) + fabsl(q) + fabsl((long double)dp);
    const long double exact = c + inc, eps = 0x1p-53L;
    if (fabsl(momentum_rhs(m, c, ew, ns, now, prev, dp) - exact) > eps * (fabsl(exact) + 6 * size)) ++far;
  }
  std::printf("moved %ld far %ld\n", moved, far);
  return moved || far;
}
