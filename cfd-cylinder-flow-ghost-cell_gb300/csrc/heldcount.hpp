// How many gated passes (refinement sweeps, Arnoldi steps) queued or captured steps hold for a solve.
#pragma once
#include <algorithm>

namespace gmk {

// A held pass that a step does not need is some kernels that return at once (2.4 us each); a step that needs
// one more than is held is repeated, with the steps queued behind it.  So the count rises with a step's
// need and falls to what a window of steps used.  Lowering a captured count means capturing again (0.3 ms a
// case), and a need that comes back doubles the window, so that a need between two counts settles on the
// larger one.  The first window is short: a first step's count is often one more than the steps behind it need
// (FP32 steps of a perturbed 96x48 grid: 202 us with what they need, 229 with two sweeps more).
struct HeldCount {
  static constexpr int FIRST = 16, WINDOW = 32, WINDOW_MAX = 4096;
  int n = 0;       // held
  int least = 0;
  int window = FIRST;
  int most = 0, seen = 0;  // the largest need of this window, its steps
  bool lowered = false;    // the last change was downwards

  void raise(int need) {
    if (need <= n) return;
    n = need;
    most = seen = 0;
    if (lowered) window = std::min(2 * window, WINDOW_MAX);
    lowered = false;
  }
  // `count` steps used at most `used` passes each; whether n changed
  bool steps(int used, int count) {
    most = std::max(most, used);
    seen += count;
    if (seen < window) return false;
    const int to = std::max(most, least);
    most = seen = 0;
    window = std::max(window, WINDOW);
    if (to >= n) return false;
    n = to;
    lowered = true;
    return true;
  }
};

}  // namespace gmk
