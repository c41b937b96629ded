// vct_cover.h -- which voxels and samples of a brick a triangle covers, in
// integer arithmetic; for the brick kernels and, compiled for the host, for
// the tests that compare the fast forms with the plain ones.
//
// Coordinates are snapped (1/256 voxel or sample) and relative to the brick.
#pragma once
#include <cstdint>
#include <type_traits>

#ifdef __CUDACC__
#define VCT_COVER_HD __host__ __device__ __forceinline__
#else
#define VCT_COVER_HD inline
#endif

namespace vct {

template <class T> VCT_COVER_HD T cover_abs(T v) { return v < 0 ? -v : v; }
template <class T> VCT_COVER_HD T cover_min(T a, T b) { return a < b ? a : b; }
template <class T> VCT_COVER_HD T cover_max(T a, T b) { return a > b ? a : b; }

VCT_COVER_HD bool axis_sep(long long p0, long long p1, long long p2, long long r) {
  return cover_min(p0, cover_min(p1, p2)) > r || cover_max(p0, cover_max(p1, p2)) < -r;
}

// Closed-box separating-axis test of triangle V against the voxel with lower
// corner 256 (x, y, z): 3 box normals, the plane, 9 edge axes.  Exact for any
// coordinates the voxelizer admits (the plane test in 128 bits).
VCT_COVER_HD bool sat_exact(const int V[3][3], int x, int y, int z) {
  const long long h = 128;
  long long u[3][3];
  const long long c[3] = {256ll * x + 128, 256ll * y + 128, 256ll * z + 128};
  for (int k = 0; k < 3; ++k)
    for (int d = 0; d < 3; ++d) u[k][d] = (long long)V[k][d] - c[d];
  for (int d = 0; d < 3; ++d)
    if (axis_sep(u[0][d], u[1][d], u[2][d], h)) return false;
  long long f[3][3];
  for (int d = 0; d < 3; ++d) {
    f[0][d] = u[1][d] - u[0][d];
    f[1][d] = u[2][d] - u[1][d];
    f[2][d] = u[0][d] - u[2][d];
  }
  const long long n0 = f[0][1] * f[1][2] - f[0][2] * f[1][1];
  const long long n1 = f[0][2] * f[1][0] - f[0][0] * f[1][2];
  const long long n2 = f[0][0] * f[1][1] - f[0][1] * f[1][0];
  const __int128 dd = (__int128)n0 * u[0][0] + (__int128)n1 * u[0][1] + (__int128)n2 * u[0][2];
  const __int128 rr = (__int128)h * ((__int128)cover_abs(n0) + (__int128)cover_abs(n1) + (__int128)cover_abs(n2));
  if (dd > rr || dd < -rr) return false;
  for (int e = 0; e < 3; ++e) {
    const long long fx = f[e][0], fy = f[e][1], fz = f[e][2];
    if (axis_sep(-fz * u[0][1] + fy * u[0][2], -fz * u[1][1] + fy * u[1][2], -fz * u[2][1] + fy * u[2][2],
                 h * (cover_abs(fz) + cover_abs(fy))))
      return false;
    if (axis_sep(fz * u[0][0] - fx * u[0][2], fz * u[1][0] - fx * u[1][2], fz * u[2][0] - fx * u[2][2],
                 h * (cover_abs(fz) + cover_abs(fx))))
      return false;
    if (axis_sep(-fy * u[0][0] + fx * u[0][1], -fy * u[1][0] + fx * u[1][1], -fy * u[2][0] + fx * u[2][1],
                 h * (cover_abs(fy) + cover_abs(fx))))
      return false;
  }
  return true;
}

// The forms of the test by the triangle's extent (1/256 voxel) along its
// longest side of the box.  Edge products stay below 2^29 (int) and the
// plane's below 2^62 (64 bits) when a vertex lies within the extent of the
// brick's 2^11.
constexpr long long kSatInt = 1ll << 13, kSatLong = 1ll << 19;

// The voxels (x, y, z0 + k), k < nz <= 8, of one column that the triangle
// touches, as bits; the same decisions as sat_exact for voxels inside the
// triangle's box (floor(min / 256 - ...) bounds: the box normals cannot
// separate there).  T = int up to kSatInt, long long up to kSatLong.
//
// On an edge's axis both its ends project to p and the third vertex to p + n
// (n: that component of the normal), so the test is one interval of p, and p
// is linear in the voxel: per further voxel an addition and a comparison for
// each of the six axes that z moves, and one for the plane.
template <class T>
VCT_COVER_HD uint32_t sat_column(const int V[3][3], int x, int y, int z0, int nz) {
  typedef typename std::make_unsigned<T>::type U;
  T u[3][3], f[3][3];
  const T c[3] = {(T)(256 * x + 128), (T)(256 * y + 128), (T)(256 * z0 + 128)};
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int d = 0; d < 3; ++d) u[k][d] = (T)V[k][d] - c[d];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    f[0][d] = u[1][d] - u[0][d];
    f[1][d] = u[2][d] - u[1][d];
    f[2][d] = u[0][d] - u[2][d];
  }
  const T n0 = f[0][1] * f[1][2] - f[0][2] * f[1][1], n1 = f[0][2] * f[1][0] - f[0][0] * f[1][2],
          n2 = f[0][0] * f[1][1] - f[0][1] * f[1][0];
  // p in [-r - max(0, n), r - min(0, n)], as 0 <= p + r + max(0, n) <= 2 r + |n|
  T lo[3][2], w[3][2];
  bool in = true;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const T fx = f[e][0], fy = f[e][1], fz = f[e][2];
    const T ax = cover_abs(fx), ay = cover_abs(fy), az = cover_abs(fz);
    const T pz = -fy * u[e][0] + fx * u[e][1] + 128 * (ax + ay) + cover_max(n2, (T)0);
    in = in & ((U)pz <= (U)(256 * (ax + ay) + cover_abs(n2)));
    lo[e][0] = -fz * u[e][1] + fy * u[e][2] + 128 * (ay + az) + cover_max(n0, (T)0);
    w[e][0] = 256 * (ay + az) + cover_abs(n0);
    lo[e][1] = fz * u[e][0] - fx * u[e][2] + 128 * (ax + az) + cover_max(n1, (T)0);
    w[e][1] = 256 * (ax + az) + cover_abs(n1);
  }
  if (!in) return 0u;
  const long long rr = 128ll * ((long long)cover_abs(n0) + cover_abs(n1) + cover_abs(n2));
  long long pl = (long long)n0 * u[0][0] + (long long)n1 * u[0][1] + (long long)n2 * u[0][2] + rr;
  uint32_t mask = 0;
#pragma unroll 1
  for (int k = 0; k < nz; ++k) {
    bool ok = (unsigned long long)pl <= (unsigned long long)(2 * rr);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      ok = ok & ((U)lo[e][0] <= (U)w[e][0]) & ((U)lo[e][1] <= (U)w[e][1]);
      lo[e][0] -= 256 * f[e][1];
      lo[e][1] += 256 * f[e][0];
    }
    pl -= 256ll * n2;
    mask |= (ok ? 1u : 0u) << k;
  }
  return mask;
}

// An edge function of the raster rule, lowered by one where the edge does not
// keep the samples on it, at the first sample of a window: floor(E / 256),
// clamped to +-2^30.  Samples are 256 apart, so E at sample (i, j) of the
// window is non-negative exactly when this + ex j - ey i is, and with i, j <
// 16 and |ex|, |ey| <= 2^25 (any coordinates the voxelizer admits) that sum
// neither overflows nor changes sign through the clamp.
VCT_COVER_HD int row_edge(long long ax, long long ay, long long bx, long long by, bool keeps, int i0, int j0) {
  const long long w = (bx - ax) * (256ll * j0 + 128 - ay) - (by - ay) * (256ll * i0 + 128 - ax) - (keeps ? 0 : 1);
  const long long lim = 1ll << 30;
  return (int)cover_max(-lim, cover_min(lim, w >> 8));
}

// The samples i < ni <= 16 of a row on which no edge is negative, as bits:
// e = the edges at its first sample, ey their steps.
VCT_COVER_HD uint32_t row_mask(int e0, int e1, int e2, int ey0, int ey1, int ey2, int ni) {
  uint32_t mask = 0;
#pragma unroll 1
  for (int i = 0; i < ni; ++i) {
    mask |= ((e0 | e1 | e2) >= 0 ? 1u : 0u) << i;
    e0 -= ey0;
    e1 -= ey1;
    e2 -= ey2;
  }
  return mask;
}

}  // namespace vct
