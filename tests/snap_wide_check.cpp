// Checks the raster's snapping over every frame extent a renderer takes
// (voxel_cone_tracing_gb300/csrc/vct_snap.h): where snap_wide lets the integer
// form run, it rounds as llrint(((double)g + 1.0) * K) does and 32 bits hold
// the coordinates and their differences.  Values near half a unit, where the
// roundings part, are tried.  Prints the faults.
#include <cmath>
#include <cstdio>
#include <random>

#include "vct_snap.h"

int main() {
  std::mt19937 rng(11);
  long long bad = 0, n = 0;
  for (int extent : {1, 771, 16383, 16384, 16385, 40000, 131071, 300000, 600001, 1 << 20, (1 << 23) + 1, 1 << 28}) {
    for (int side = 0; side < 2; ++side) {
      if (side ? vct::snap_wide(extent, 1) : vct::snap_wide(1, extent)) continue;
      const double K = extent * 128.0;
      if (64.0 * 2 * K >= 2147483647.0) ++bad;
      std::uniform_real_distribution<double> wide(-64.0 * K, 64.0 * K);
      for (int i = 0; i < 200000; ++i) {
        const float g = (float)((std::floor(wide(rng)) + 0.5) / K - 1.0);
        for (float v : {g, std::nextafter(g, 99.f), std::nextafter(g, -99.f)}) {
          if (!(std::fabs(v) <= 64.f)) continue;
          bool close;
          const int got = vct::snap_scaled(v, (uint32_t)K, close);
          ++n;
          if (!close && got != std::llrint(((double)v + 1.0) * K)) ++bad;
        }
      }
    }
  }
  std::printf("%lld of %lld wrong\n", bad, n);
  return bad != 0;
}
