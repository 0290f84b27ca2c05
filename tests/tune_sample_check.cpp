// Host check of the autotuner's sample: both streams' polys of a batch-sized
// call lie inside the buffer, as does the whole sample.
#include <cstdio>

#include "../aoa_b200/csrc/tune_sample.h"

int main() {
  for (int log_n = 10; log_n <= 17; log_n++)
    for (int k = 1; k <= 64; k++)
      for (long limbs = 0; limbs <= 40 * k; limbs++) {
        const aoa::TuneSample s = aoa::tune_sample(limbs, k, 1L << log_n);
        if (s.npolys < 1 || s.half < 1 || s.npolys * k < limbs || s.polys < s.npolys || s.polys < 2L * s.half) {
          std::printf("log_n %d k %d limbs %ld: %ld polys, half %d, buffer %ld\n", log_n, k, limbs, s.npolys, s.half,
                      s.polys);
          return 1;
        }
      }
  std::printf("ok\n");
  return 0;
}
