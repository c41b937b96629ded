// vct_snap.h -- exact fixed-point snapping of FP32 grid-space coordinates,
// in integer arithmetic (host and device).
//
// The voxelizers snap each vertex coordinate g (grid space, |g| <= 64) to
// round((g + 1) * 2^k), rounding half to even, with 2^k = N * 256 (the 2N x
// 2N raster's 1/256-sample grid) or N * 128 (the conservative rule's 1/256
// voxel).  The result is the exact value of that expression: g = m * 2^e
// with a 24-bit integer m, so (g + 1) * 2^k = 2^k + m * 2^(e + k); the
// second term is an integer or is rounded half to even by a shift, and
// adding the even integer 2^k does not change which neighbour is even.
// (It equals rounding the double (double)g + 1.0 scaled by 2^k: that sum is
// exact for |g| >= 2^-29, and for smaller g both give 2^k.)  No FP64
// arithmetic is involved.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define VCT_SNAP_HD __host__ __device__
#else
#define VCT_SNAP_HD
#endif

namespace vct {

// round-half-even((g + 1) * 2^k) for finite g with |g| <= 64 and 1 <= k <= 24.
VCT_SNAP_HD inline long long snap_fixed(float g, int k) {
#ifdef __CUDA_ARCH__
  const uint32_t bits = __float_as_uint(g);
#else
  uint32_t bits;
  std::memcpy(&bits, &g, sizeof(bits));
#endif
  const int exp = (int)((bits >> 23) & 0xffu);
  const long long base = 1LL << k;
  if (exp == 0) return base;  // zero or subnormal: |g * 2^k| < 1/2
  const uint32_t m = (bits & 0x7fffffu) | 0x800000u;
  const int s = exp - 150 + k;  // g * 2^k = m * 2^s
  long long q;
  if (s >= 0) {
    q = (long long)m << s;
  } else {
    const int sh = -s;
    if (sh > 24) {
      q = 0;  // m * 2^s < 1/2
    } else {
      const uint32_t rem = m & ((1u << sh) - 1u), half = 1u << (sh - 1);  // sh in [1, 24]
      q = (long long)(m >> sh);
      if (rem > half || (rem == half && (q & 1))) ++q;
    }
  }
  return (bits >> 31) ? base - q : base + q;
}

// round-half-even((g + 1) * K) as FP64 computes it -- the sum and the product
// each rounded once -- for |g| <= 64 and 1 <= K <= 2^21 (K need not be a power
// of two: 128 times a frame's width or height).  With g = m * 2^-s the exact
// value is K + m K / 2^s, m K below 2^45; FP64's own rounding moves it by less
// than 2^-24, so an integer shift rounds alike unless the fraction is that near
// one half.  `close` reports such a value (and returns nothing of use): the
// caller then rounds in FP64.  A frame wider or higher than kSnapPixels is
// snapped in FP64 throughout (snap_wide): there FP64's own rounding reaches
// past that band, and coordinates and their differences past 32 bits.
constexpr int kSnapPixels = 1 << 14;
inline bool snap_wide(int W, int H) { return W > kSnapPixels || H > kSnapPixels; }
VCT_SNAP_HD inline int snap_scaled(float g, uint32_t K, bool& close) {
#ifdef __CUDA_ARCH__
  const uint32_t bits = __float_as_uint(g);
#else
  uint32_t bits;
  std::memcpy(&bits, &g, sizeof(bits));
#endif
  close = false;
  const int exp = (int)((bits >> 23) & 0xffu);
  if (exp < 127 - 31) return (int)K;  // |g K| < 2^-10
  const long long m = (long long)((bits & 0x7fffffu) | 0x800000u) * K;
  const long long p = (bits >> 31) ? -m : m;
  const int s = 150 - exp;  // in [17, 54]
  const long long half = 1LL << (s - 1);
  const long long off = (p & ((1LL << s) - 1)) - half;  // the fraction's distance from one half
  const long long band = s > 24 ? 1LL << (s - 24) : 0;
  close = off <= band && off >= -band;
  return (int)K + (int)((p + half) >> s);
}

}  // namespace vct
