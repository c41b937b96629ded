// Checks voxel_cone_tracing_gb300/csrc/vct_tiles.h: a box's tiles cover it
// once, no other tile number gives an origin, however far past the box, and
// counts of records and tiles stay apart.  Prints the faults found.
#include <cstdio>
#include <random>
#include <vector>

#include "vct_tiles.h"

int main() {
  using namespace vct;
  std::mt19937_64 rng(5);
  long long bad = 0;
  for (int i = 0; i < 400; ++i) {
    const int W = 1 + (int)(rng() % (i % 4 ? 200 : 16384)), H = 1 + (int)(rng() % (i % 4 == 1 ? 16384 : 200));
    int x0 = (int)(rng() % W), x1 = (int)(rng() % W), y0 = (int)(rng() % H), y1 = (int)(rng() % H);
    if (x0 > x1) std::swap(x0, x1);
    if (y0 > y1) std::swap(y0, y1);
    const uint32_t across = tiles_across(x0, x1), n = tiles_of(x0, y0, x1, y1);
    std::vector<int> seen((size_t)n, 0);
    for (uint32_t t = 0; t < n; ++t) {
      int px = -1, py = -1;
      if (!tile_origin(t, across, x0, y0, y1, px, py) || px < x0 || px > x1 || py < y0 || py > y1 ||
          (px - x0) % kTile || (py - y0) % kTile)
        ++bad;
      else
        ++seen[(size_t)(py - y0) / kTile * across + (px - x0) / kTile];
    }
    for (int s : seen) bad += s != 1;
    int px, py;
    for (int k = 0; k < 64; ++k) {  // past the box: just, by 2^26 rows (a row's 32 pixels pass 2^31), by 2^32 tiles
      const unsigned long long far[] = {n + k, (unsigned long long)across * ((1u << 26) - 32 + k), (1ull << 31) + k,
                                        (1ull << 32) - 1 - k, (1ull << 32) + k, (1ull << 33) + rng() % n};
      for (unsigned long long t : far)
        if (t >= n) bad += tile_origin(t, across, x0, y0, y1, px, py);
    }
  }
  // 65,000 triangles that fill 16384x16384 pixels, then a million of one tile
  unsigned long long count = 0, tiles = 0;
  for (uint32_t i = 0; i < 65000; ++i) {
    bad += big_records(count) != i || big_tiles(count) != tiles;
    const uint32_t t = tiles_of(0, 0, 16383, 16383);
    count += big_count_of(1, t);
    tiles += t;
  }
  count += big_count_of(1, 1) * 1000000u;
  bad += big_records(count) != 1065000u || big_tiles(count) != tiles + 1000000u;
  std::printf("%lld faults\n", bad);
  return bad != 0;
}
