// The polys that the autotuner's timings work on (host code; tune.cu).
#pragma once
#include <algorithm>

namespace aoa {

struct TuneSample {
  long npolys;   // polys of the whole-sample calls
  int half;      // polys of a batch-sized call, on each of two streams side by side
  long polys;    // polys of the buffer
};

// limbs > 0: a sample of that many limbs, 0: about 12x the L2 size, in whole polys of k limbs
inline TuneSample tune_sample(long limbs, int k, long N) {
  const long want = limbs > 0 ? limbs : std::max<long>(k, (1536L << 20) / (8 * N));
  TuneSample s;
  s.npolys = std::max<long>(1, (want + k - 1) / k);
  s.half = (int)std::max(1L, std::min(s.npolys / 2, 8L));
  s.polys = std::max(s.npolys, 2L * s.half);   // a sample of one poly has a second stream's beside it
  return s;
}

}  // namespace aoa
