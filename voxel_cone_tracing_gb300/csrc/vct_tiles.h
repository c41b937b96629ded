// vct_tiles.h -- the tiles of the G-buffer raster's large triangles: how they
// are counted and where one lies; for the raster's kernels and, compiled for
// the host, for their test.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define VCT_TILES_HD __host__ __device__ __forceinline__
#else
#define VCT_TILES_HD inline
#endif

namespace vct {

constexpr int kTileBits = 5;  // a large triangle's tile: 32x32 pixels of its box
constexpr int kTile = 1 << kTileBits;

// Records and tiles are counted in one 64-bit word, so that the first tiles
// ascend with the records.  Tiles take the low 34 bits (65,000 triangles that
// fill 16384x16384 pixels, 8.4 million at 1920x1080), records the other 30
// (their triangles alone would fill the device's memory); with 32 and 32 the
// tiles of 2.1 million full 1920x1080 screens ran over into the records.
constexpr int kTileCountBits = 34;
VCT_TILES_HD unsigned long long big_count_of(unsigned long long records, unsigned long long tiles) {
  return records << kTileCountBits | tiles;
}
VCT_TILES_HD uint32_t big_records(unsigned long long count) { return (uint32_t)(count >> kTileCountBits); }
VCT_TILES_HD unsigned long long big_tiles(unsigned long long count) {
  return count & ((1ull << kTileCountBits) - 1ull);
}

// Tiles across and in all of the box [x0, x1] x [y0, y1] (pixels, inclusive).
VCT_TILES_HD uint32_t tiles_across(int x0, int x1) { return (uint32_t)(x1 - x0 + kTile) >> kTileBits; }
VCT_TILES_HD uint32_t tiles_of(int x0, int y0, int x1, int y1) {
  return tiles_across(x0, x1) * tiles_across(y0, y1);
}

// The first pixel of tile t of the box; false for a t that the box does not
// have (past a full list's last record).
VCT_TILES_HD bool tile_origin(unsigned long long t, uint32_t across, int x0, int y0, int y1, int& px, int& py) {
  if (t >= 1ull << 32) return false;
  const uint32_t row = (uint32_t)t / across;
  if (row >= tiles_across(y0, y1)) return false;
  px = x0 + (int)((uint32_t)t - row * across) * kTile;
  py = y0 + (int)row * kTile;
  return true;
}

}  // namespace vct
