// Checks vct::snap_scaled (voxel_cone_tracing_gb300/csrc/vct_snap.h) against
// llrint(((double)g + 1.0) * K), the FP64 rounding it replaces, for K = 128
// times frame extents from 1 to 16384.  Prints the mismatches among the values
// it decides and, of the evenly spread ones, how many it leaves to FP64.
#include <cmath>
#include <cstdio>
#include <random>

#include "vct_snap.h"

int main() {
  std::mt19937 rng(3);
  long long bad = 0, n = 0, spread = 0, left = 0;
  for (int extent : {1, 2, 3, 17, 37, 320, 771, 1080, 1367, 1920, 4096, 5000, 16383, 16384}) {
    const int K = extent * 128;
    auto check = [&](float g) {
      bool close;
      const int v = vct::snap_scaled(g, (uint32_t)K, close);
      ++n;
      if (!close && v != std::llrint(((double)g + 1.0) * (double)K)) ++bad;
      return close;
    };
    std::uniform_real_distribution<float> wide(-64.f, 64.f), unit(-1.5f, 1.5f);
    std::uniform_real_distribution<double> tiny(-45.0, 0.0);
    for (int i = 0; i < 100000; ++i) {
      left += check(wide(rng));
      left += check(unit(rng));
      spread += 2;
      check((float)std::ldexp(1.0, (int)tiny(rng)) * unit(rng));
    }
    for (int j = -5000; j < 5000; ++j) {  // halves and their neighbours
      const float g = (float)((j + 0.5) / K - 1.0);
      check(g);
      check(std::nextafter(g, 9.f));
      check(std::nextafter(g, -9.f));
    }
    for (float g : {0.f, -0.f, 1e-40f, -1e-40f, 0x1p-31f, 0x1p-32f, -0x1p-31f, 64.f, -64.f, 1.f, -1.f, .5f, -.5f})
      check(g);
  }
  std::printf("%lld of %lld differ, %lld of %lld left\n", bad, n, left, spread);
  return bad != 0;
}
