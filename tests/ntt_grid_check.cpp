// Host check of a transform pass's grid: a chosen number of waves is what is
// launched (to a group of tile columns), whatever the call's size; no CTA is
// without work and one exists for every tile column.
#include <cstdio>

#include "../aoa_b200/csrc/ntt_grid.h"

int main() {
  for (int resident : {148, 296, 444, 592})
    for (int tiles = 1; tiles <= 512; tiles *= 2)
      for (int items = 1; items <= 3000; items += 1 + items / 8)
        for (double waves : {0.01, 0.5, 1.0, 2.0, 2.5, 8.0, 64.0})
          for (double def : {1.0, 8.0}) {
            const int share = 1 + items % 5;
            const int g = aoa::ctas_per_tile(waves, def, share, resident, tiles, items);
            const double want = waves * resident / tiles;   // CTAs per tile column of that many waves
            const double mean = (double)items * tiles / resident;
            const bool each = g == items, wave = (g == 1 || g <= want) && (each || g + 1 > want);
            bool ok = g >= 1 && g <= items && (wave || (each && waves == def && mean <= 2.5));
            if (waves == def && (share == 1 ? mean <= 2.5 : share > 3 && mean <= 1.2)) ok = ok && each;
            if (!ok) {
              std::printf("waves %g (default %g), resident %d, tiles %d, items %d: %d\n", waves, def, resident, tiles,
                          items, g);
              return 1;
            }
          }
  std::printf("ok\n");
  return 0;
}
