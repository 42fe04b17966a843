// How many gated passes (refinement sweeps, Arnoldi steps) queued or captured steps hold for a solve.
#pragma once
#include <algorithm>

namespace gmk {

// A held pass that a step does not need is some kernels that return at once (2.4 us each); a step that needs
// one more than is held is repeated, with the steps queued behind it.  So the count rises with a step's
// need and falls to what a window of steps used.  Lowering a captured count means capturing again, and
// a need that comes back doubles the window, so that a need between two counts settles on the larger one.
struct HeldCount {
  int n = 0;       // held
  int least = 0;
  int window = 64;
  int most = 0, seen = 0;  // the largest need of this window, its steps
  bool lowered = false;    // the last change was downwards

  void raise(int need) {
    if (need <= n) return;
    n = need;
    most = seen = 0;
    if (lowered) window = std::min(2 * window, 4096);
    lowered = false;
  }
  // `count` steps used at most `used` passes each; whether n changed
  bool steps(int used, int count) {
    most = std::max(most, used);
    seen += count;
    if (seen < window) return false;
    const int to = std::max(most, least);
    most = seen = 0;
    if (to >= n) return false;
    n = to;
    lowered = true;
    return true;
  }
};

}  // namespace gmk
