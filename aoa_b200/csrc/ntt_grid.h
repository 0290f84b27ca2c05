// Grid of a transform pass (host code; the launchers of ntt_kernels.cuh).
#pragma once
#include <algorithm>

namespace aoa {

// CTAs per tile column of a pass over `items` limbs of `tiles` tiles each, with
// `resident` CTAs on the chip at once: about `waves` of those (a knob), each
// looping over its limbs.  At the knob's default, calls of up to two and a half
// waves run one tile per CTA: with one wave of CTAs some of them hold two tiles
// and some three (31 limbs in 27 groups at 2^16: two for 4 groups, one for 23),
// and the pass ends with the longest.
inline int ctas_per_tile(double waves, double default_waves, int resident, int tiles, int items) {
  if (waves == default_waves && (double)items * tiles <= 2.5 * resident) return items;
  const int target = std::max(1, (int)(waves * resident) / std::max(1, tiles));
  return std::max(1, std::min(items, target));
}

}  // namespace aoa
