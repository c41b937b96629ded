// Checks the brick kernels' coverage forms (voxel_cone_tracing_gb300/csrc/
// vct_cover.h) against the plain ones: sat_column<int> and <long long> against
// sat_exact on every voxel of a triangle's box in a brick, and row_edge /
// row_mask against the 64-bit edge functions with their fill rule on every
// sample of a window.  Prints the differences and exits non-zero on any.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "vct_cover.h"

static long long bad = 0, voxels = 0, touched = 0, samples = 0, inside = 0;

static void columns(const int V[3][3], bool fits_int) {
  int lo[3], hi[3];
  for (int d = 0; d < 3; ++d) {
    const int mn = std::min({V[0][d], V[1][d], V[2][d]}), mx = std::max({V[0][d], V[1][d], V[2][d]});
    lo[d] = std::max(0, ((mn + 255) >> 8) - 1);
    hi[d] = std::min(7, mx >> 8);
    if (hi[d] < lo[d]) return;
  }
  for (int y = lo[1]; y <= hi[1]; ++y)
    for (int x = lo[0]; x <= hi[0]; ++x) {
      const int nz = hi[2] - lo[2] + 1;
      uint32_t want = 0;
      for (int k = 0; k < nz; ++k) want |= (vct::sat_exact(V, x, y, lo[2] + k) ? 1u : 0u) << k;
      bad += vct::sat_column<long long>(V, x, y, lo[2], nz) != want;
      if (fits_int) bad += vct::sat_column<int>(V, x, y, lo[2], nz) != want;
      voxels += nz;
      touched += __builtin_popcount(want);
    }
}

static void rows(const long long X[3], const long long Y[3]) {
  bool keeps[3];
  for (int k = 0; k < 3; ++k) keeps[k] = (X[k] + Y[k] + k) & 1;  // any fill rule
  const int i0 = 3, j0 = 2, ni = 13, nj = 14;
  int e[3], ex[3], ey[3];
  for (int k = 0; k < 3; ++k) {
    const int a = (k + 1) % 3, b = (k + 2) % 3;
    e[k] = vct::row_edge(X[a], Y[a], X[b], Y[b], keeps[k], i0, j0);
    ex[k] = (int)(X[b] - X[a]);
    ey[k] = (int)(Y[b] - Y[a]);
  }
  for (int j = 0; j < nj; ++j) {
    uint32_t want = 0;
    for (int i = 0; i < ni; ++i) {
      bool in = true;
      for (int k = 0; k < 3; ++k) {
        const int a = (k + 1) % 3, b = (k + 2) % 3;
        const __int128 w = (__int128)(X[b] - X[a]) * (256 * (j0 + j) + 128 - Y[a]) -
                           (__int128)(Y[b] - Y[a]) * (256 * (i0 + i) + 128 - X[a]);
        in = in && (w > 0 || (w == 0 && keeps[k]));
      }
      want |= (in ? 1u : 0u) << i;
    }
    bad += vct::row_mask(e[0] + ex[0] * j, e[1] + ex[1] * j, e[2] + ex[2] * j, ey[0], ey[1], ey[2], ni) != want;
    samples += ni;
    inside += __builtin_popcount(want);
  }
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 20000;
  std::mt19937 rng(11);
  auto in = [&](long long lo, long long hi) { return std::uniform_int_distribution<long long>(lo, hi)(rng); };
  for (long i = 0; i < n; ++i) {
    // extents from a sixteenth of a voxel to the widest of each form; a third
    // on voxel corners, edges and centres; some flat, collinear or a point
    const long long ext = 1ll << (i % 20);
    int V[3][3];
    for (int d = 0; d < 3; ++d) {
      const long long at = in(-ext, 2048);
      for (int k = 0; k < 3; ++k) {
        long long v = at + in(0, ext);
        if (i % 3 == 0) v = std::min((v + 64) / 128 * 128, at / 128 * 128 + ext);
        V[k][d] = (int)v;
      }
    }
    if (i % 7 == 0) V[1][i % 3] = V[0][i % 3], V[2][i % 3] = V[0][i % 3];
    if (i % 11 == 0) for (int d = 0; d < 3; ++d) V[2][d] = V[1][d];
    if (i % 13 == 0) for (int d = 0; d < 3; ++d) V[2][d] = 2 * V[1][d] - V[0][d] > (1 << 20) ? V[0][d] : V[1][d];
    long long widest = 0;
    for (int d = 0; d < 3; ++d)
      widest = std::max(widest, (long long)std::max({V[0][d], V[1][d], V[2][d]}) - std::min({V[0][d], V[1][d], V[2][d]}));
    if (widest <= vct::kSatLong) columns(V, widest <= vct::kSatInt);

    const long long side = 1ll << (4 + i % 22);  // up to 2^25
    long long X[3], Y[3];
    const long long ox = in(-side, 4096), oy = in(-side, 4096);
    for (int k = 0; k < 3; ++k) {
      X[k] = ox + in(0, side);
      Y[k] = oy + in(0, side);
      if (i % 4 == 0) X[k] = X[k] / 256 * 256 + 128, Y[k] = Y[k] / 256 * 256 + 128;
      X[k] = std::min(X[k], ox + side);
      Y[k] = std::min(Y[k], oy + side);
    }
    if ((X[1] - X[0]) * (Y[2] - Y[0]) < (Y[1] - Y[0]) * (X[2] - X[0])) std::swap(X[1], X[2]), std::swap(Y[1], Y[2]);
    rows(X, Y);
  }
  std::printf("%lld differ; %lld of %lld voxels, %lld of %lld samples covered\n", bad, touched, voxels, inside, samples);
  return bad != 0;
}
