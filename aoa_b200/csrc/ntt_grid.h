// Grid of a transform pass (host code; the launchers of ntt_kernels.cuh).
#pragma once
#include <algorithm>

namespace aoa {

// CTAs per tile column of a pass over `items` limbs of `tiles` tiles each, with
// `resident` CTAs on the chip at once: about `waves` of those (a knob), each
// looping over its limbs.
//
// At the knob's default, calls of up to two and a half waves may run one tile
// per CTA: with one wave of CTAs some of them hold two tiles and some three (31
// limbs in 27 groups at 2^16: two for 4 groups, one for 23), and the pass ends
// with the longest.  The column pass always does (us of a transform, one wave ->
// a CTA per tile, primes q = 1 mod 2^32: 36 limbs of 2^16 (1.30 waves) 39.1 ->
// 35.8 forward, 41.1 -> 36.5 inverse, 68 (2.45) 60.7 -> 59.9 and 62.7 -> 61.0; 34
// of 2^17 105.9 -> 95.5; 240 of 2^14 (2.16) 57.1 -> 52.4), and so does a row pass of
// one poly (17 limbs of 2^16 (1.23) 24.6 -> 21.4, 31 (2.23) 36.6 -> 35.1).  A row
// pass that holds the next poly under the same prime keeps its twiddles: with two
// or three polys it loops unless the longest CTA would hold 1.3 times the mean (two
// polys: 20 limbs of 2^16 (1.44) 24.2 -> 23.6, 22 (1.59) 24.3 -> 25.2; 38 of 2^15
// (1.37) 25.5 -> 23.6, 50 (1.80) 26.2 -> 28.3; HMult at 2^15 whose inverse has 54
// limbs 151.9 -> 157.7, 58 limbs 126.5 -> 124.5), with more from
// 1.2 waves on (eight: 32 limbs of 2^15 (1.15) 23.4 -> 22.0, 40 (1.44) 24.0 -> 26.5,
// 64 (2.31) 33.0 -> 37.9).
// share: polys under a prime whose tables the pass keeps (1 for the column pass).
inline int ctas_per_tile(double waves, double default_waves, int share, int resident, int tiles, int items) {
  const int target = std::max(1, (int)(waves * resident) / std::max(1, tiles));
  const double mean = (double)items * tiles / resident;
  if (waves == default_waves && mean <= 2.5) {
    const int groups = std::max(1, resident / std::max(1, tiles)), longest = (items + groups - 1) / groups;
    if (share == 1 || (share <= 3 ? longest > 1.3 * mean : mean <= 1.2)) return items;
  }
  return std::max(1, std::min(items, target));
}

}  // namespace aoa
