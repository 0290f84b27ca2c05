// Grid of a transform pass (host code; the launchers of ntt_kernels.cuh).
#pragma once
#include <algorithm>

namespace aoa {

// CTAs per tile column of a pass over `items` limbs of `tiles` tiles each, with
// `resident` CTAs on the chip at once: about `waves` of those (a knob), each
// looping over its limbs.  At the knob's default, calls of up to `apart` waves
// run one tile per CTA: with one wave of CTAs some of them hold two tiles and
// some three (31 limbs in 27 groups at 2^16: two for 4 groups, one for 23), and
// the pass ends with the longest.
inline int ctas_per_tile(double waves, double default_waves, double apart, int resident, int tiles, int items) {
  if (waves == default_waves && (double)items * tiles <= apart * resident) return items;
  const int target = std::max(1, (int)(waves * resident) / std::max(1, tiles));
  return std::max(1, std::min(items, target));
}

// `apart` of the two passes.  Of the column pass at any call up to 2.5 waves
// (us of a transform, one wave -> a CTA per tile, primes q = 1 mod 2^32: 36 limbs
// of 2^16 (1.30 waves) 39.1 -> 35.8 forward, 41.1 -> 36.5 inverse, 68 (2.45) 60.7
// -> 59.9 and 62.7 -> 61.0; 34 of 2^17 105.9 -> 95.5; 240 of 2^14 (2.16) 57.1 ->
// 52.4).  A row pass that holds the next poly under the same prime keeps its
// twiddles, which soon is worth more than the even end.  One poly: 17 limbs of 2^16
// (1.23) 24.6 -> 21.4, 31 (2.23) 36.6 -> 35.1.  Two: 20 limbs of 2^16 (1.44) 24.2 ->
// 23.6, 22 (1.59) 24.3 -> 25.2; 38 of 2^15 (1.37) 25.5 -> 23.6, 50 (1.80) 26.2 ->
// 28.3.  Eight: 32 of 2^15 (1.15) 23.4 -> 22.0, 40 (1.44) 24.0 -> 26.5, 64 (2.31)
// 33.0 -> 37.9.
inline double cols_apart() { return 2.5; }
inline double rows_apart(int npolys) { return npolys == 1 ? 2.5 : npolys <= 3 ? 1.5 : 1.2; }

}  // namespace aoa
