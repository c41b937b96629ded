// vct_cone.cuh -- the pieces of the ConeTracer that its kernels share
// (k_trace.cu, k_trace_frame.cu): the samplers, the cone marches, the diffuse
// cones' directions, far-field groups and lights of voxel_cone_tracing.frag.
//
// The files that include it are compiled with -fmad=false: a product and a
// sum are fused only where the code says so (__fmaf_rn), so the results do
// not depend on how the compiler arranges the code around them.
//
// Texture sampling is GL textureLod with GL_LINEAR_MIPMAP_LINEAR and
// CLAMP_TO_BORDER(0) over levels 0..L-1 (texture_3d.cpp:10-15).  Level 0 is
// one texture shared by the six maps (as in the reference, where all six
// maps hold identical level-0 data), so for lambda < 1 the three per-axis
// lookups of sample_voxel (:80-86) need one level-0 fetch:
//   sum_k a_k [(1-f) T0 + f T1_k] = (1-f) T0 sum_k a_k + f sum_k a_k T1_k.
// Two samplers:
//   VCT_SAMPLER_HW    -- the texture unit filters (trilinear within a level,
//                        linear between levels; 8-bit fixed-point weights);
//   VCT_SAMPLER_EXACT -- FP32 trilinear / mip-linear filtering in software
//                        from surface reads (the accuracy reference).
#pragma once

#include <cuda_fp16.h>

#include <type_traits>

#include "vct_internal.h"
#include "vct_math.cuh"

namespace vct {
namespace {

#define VCT_STR(x) #x
#define VCT_UNROLL_N(n) _Pragma(VCT_STR(unroll n))

__device__ __forceinline__ float4 f4(float x, float y, float z, float w) { return make_float4(x, y, z, w); }
__device__ __forceinline__ float4 operator+(float4 a, float4 b) { return f4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 operator*(float4 a, float s) { return f4(a.x * s, a.y * s, a.z * s, a.w * s); }
// a * s and a * s + c with one rounding each, spelled out so that the alpha
// channel is computed identically by the RGBA and the alpha-only paths.
__device__ __forceinline__ float4 mul4(float4 a, float s) {
  return f4(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s), __fmul_rn(a.w, s));
}
__device__ __forceinline__ float4 fma4(float4 a, float s, float4 c) {
  return f4(__fmaf_rn(a.x, s, c.x), __fmaf_rn(a.y, s, c.y), __fmaf_rn(a.z, s, c.z), __fmaf_rn(a.w, s, c.w));
}

constexpr float kTan22_5 = 0.55785173935f;      // TAN_22_5 (:136), kept verbatim
constexpr float kMaxDistance = 1.73205080757f;  // MAX_DISTANCE (:138)
constexpr float kSixAperture = 1.15470053838f;  // 2 tan(30 deg)

// ---------------------------------------------------------------- samplers --
template <int STORAGE>
__device__ __forceinline__ float4 fetch_texel(cudaSurfaceObject_t s, int x, int y, int z) {
  if (STORAGE == VCT_STORAGE_RGBA8) {
    unsigned v;
    surf3Dread(&v, s, x * 4, y, z, cudaBoundaryModeZero);
    // a byte as a float: the low bits of 2^23 + byte
    const float k = 1.0f / 255.0f, b = 8388608.0f;
    return f4((__uint_as_float(__byte_perm(v, 0x4b000000u, 0x7440)) - b) * k,
              (__uint_as_float(__byte_perm(v, 0x4b000000u, 0x7441)) - b) * k,
              (__uint_as_float(__byte_perm(v, 0x4b000000u, 0x7442)) - b) * k,
              (__uint_as_float(__byte_perm(v, 0x4b000000u, 0x7443)) - b) * k);
  } else {
    uint2 v;
    surf3Dread(&v, s, x * 8, y, z, cudaBoundaryModeZero);
    const float2 a = __half22float2(*reinterpret_cast<__half2*>(&v.x));
    const float2 b = __half22float2(*reinterpret_cast<__half2*>(&v.y));
    return f4(a.x, a.y, b.x, b.y);
  }
}

__device__ __forceinline__ bool u_sane(V3 u) {
  return fabsf(u.x) < 1.0e6f && fabsf(u.y) < 1.0e6f && fabsf(u.z) < 1.0e6f;
}

// sum_k a_k * textureLod(map idx_k, u, lod) in FP32: trilinear within a level
// (texels outside are 0), linear between levels.  The three maps of a level
// are filtered together: their corners and weights are the same, and so are
// their texels at level 0.
template <bool ISO, int STORAGE>
__device__ __forceinline__ float4 sample_exact(const MapSet& m, V3 u, int ix, int iy, int iz, V3 ad, float lod) {
  constexpr int K = ISO ? 1 : 3;
  if (!u_sane(u)) return f4(0.f, 0.f, 0.f, 0.f);
  const int q = m.L - 1;
  int level = 0;
  float f = 0.0f;  // > 0: also level + 1
  bool two = false;
  if (lod >= (float)q) {
    level = q;
  } else if (lod > 0.0f) {
    const float fl = floorf(lod);
    level = (int)fl;
    f = lod - fl;
    two = true;
  }
  float4 r[K];
#pragma unroll 1
  for (int j = 0; j < (two ? 2 : 1); ++j, ++level) {
    const int s = m.N >> level;
    const float tx = u.x * (float)s - 0.5f, ty = u.y * (float)s - 0.5f, tz = u.z * (float)s - 0.5f;
    const float fx = floorf(tx), fy = floorf(ty), fz = floorf(tz);
    const float ax = tx - fx, ay = ty - fy, az = tz - fz;
    const int cx = (int)fx, cy = (int)fy, cz = (int)fz;
    float4 t[K];
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] = f4(0.f, 0.f, 0.f, 0.f);
    cudaSurfaceObject_t surf[K];
    surf[0] = level == 0 ? m.l0_surf : m.surf[ISO ? 0 : ix][level];
    if constexpr (!ISO) {
      surf[1] = m.surf[iy][level];
      surf[2] = m.surf[iz][level];
    }
#pragma unroll 2
    for (int c = 0; c < 8; ++c) {
      const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
      const float w = (dx ? ax : 1.0f - ax) * (dy ? ay : 1.0f - ay) * (dz ? az : 1.0f - az);
      const int X = cx + dx, Y = cy + dy, Z = cz + dz;
      // (the surface would return 0 outside, but slower: 692 -> 883 us)
      if ((unsigned)X < (unsigned)s && (unsigned)Y < (unsigned)s && (unsigned)Z < (unsigned)s) {
        t[0] = t[0] + fetch_texel<STORAGE>(surf[0], X, Y, Z) * w;
        if (!ISO && level > 0) {
#pragma unroll
          for (int k = 1; k < K; ++k) t[k] = t[k] + fetch_texel<STORAGE>(surf[k], X, Y, Z) * w;
        }
      }
    }
    if (level == 0) {
#pragma unroll
      for (int k = 1; k < K; ++k) t[k] = t[0];
    }
#pragma unroll
    for (int k = 0; k < K; ++k) r[k] = j ? r[k] + t[k] * f : (two ? t[k] * (1.0f - f) : t[k]);
  }
  if constexpr (ISO) return r[0] * (ad.x + ad.y + ad.z);
  else return r[0] * ad.x + r[1] * ad.y + r[2] * ad.z;
}

// sum_k a_k * textureLod(chain idx_k, u, l) from the texture unit.  A map
// whose weight is exactly 0 is not fetched: its term 0 * texel is 0 for every
// finite texel, so the sum is unchanged.  Cones along an axis-aligned normal
// (every wall pixel) have one or two such weights.
// One map of an axis, the negative (D) or the positive (D + 1) one.  FIXED:
// two fetches with handles at fixed addresses, of which each lane takes one;
// else the lane's handle is looked up.  The look-up costs instructions (the
// first samples of k_shade, which are bound by those, ran 177 -> 160 us on
// the bench frame with FIXED), the pair costs the texture unit partly filled
// quads (7% more filter wavefronts: what the marches are bound by).
template <int D, bool FIXED>
__device__ __forceinline__ float4 axis_fetch(const MapSet& m, V3 u, bool positive, float l) {
  if constexpr (!FIXED) return tex3DLod<float4>(m.tex[positive ? D + 1 : D], u.x, u.y, u.z, l);
  if (positive) return tex3DLod<float4>(m.tex[D + 1], u.x, u.y, u.z, l);
  return tex3DLod<float4>(m.tex[D], u.x, u.y, u.z, l);
}

// Which map of each axis a direction samples (-1 or +1 side), one word.
// again(): the same word, opaque to the compiler, so that a loop looks the
// handles up from it at every step instead of holding six registers of them.
__device__ __forceinline__ int octant(V3 d) {
  return (d.x < 0.0f ? 0 : 1) | (d.y < 0.0f ? 0 : 2) | (d.z < 0.0f ? 0 : 4);
}
__device__ __forceinline__ int again(int oct) {
  asm volatile("" : "+r"(oct));
  return oct;
}

// (not FIXED: any map for any axis, as the voxel debug view asks for)
template <bool FIXED>
__device__ __forceinline__ float4 aniso_fetch(const MapSet& m, V3 u, int ix, int iy, int iz, V3 ad, float l) {
  auto fetch = [&](auto axis, int i) {
    if constexpr (FIXED) return axis_fetch<decltype(axis)::value, true>(m, u, i != decltype(axis)::value, l);
    else return tex3DLod<float4>(m.tex[i], u.x, u.y, u.z, l);
  };
  float4 r = f4(0.f, 0.f, 0.f, 0.f);
  if (ad.x != 0.0f) r = mul4(fetch(std::integral_constant<int, 0>(), ix), ad.x);
  if (ad.y != 0.0f) r = fma4(fetch(std::integral_constant<int, 2>(), iy), ad.y, r);
  if (ad.z != 0.0f) r = fma4(fetch(std::integral_constant<int, 4>(), iz), ad.z, r);
  return r;
}

// The alpha channel of aniso_fetch from the alpha chain of the direction's x
// and y signs (MapSet::alpha_tex).  The texture unit filters every channel
// with the same weights, so each term equals the alpha of the corresponding
// map's fetch bit for bit; a map of weight 0 adds nothing.
template <bool FIXED>
__device__ __forceinline__ float4 alpha_fetch(const MapSet& m, V3 u, V3 dir, float l) {
  if constexpr (!FIXED)
    return tex3DLod<float4>(m.alpha_tex[(dir.x < 0.0f ? 0 : 1) + (dir.y < 0.0f ? 0 : 2)], u.x, u.y, u.z, l);
  if (dir.x < 0.0f) {
    if (dir.y < 0.0f) return tex3DLod<float4>(m.alpha_tex[0], u.x, u.y, u.z, l);
    return tex3DLod<float4>(m.alpha_tex[2], u.x, u.y, u.z, l);
  }
  if (dir.y < 0.0f) return tex3DLod<float4>(m.alpha_tex[1], u.x, u.y, u.z, l);
  return tex3DLod<float4>(m.alpha_tex[3], u.x, u.y, u.z, l);
}
__device__ __forceinline__ float combine_alpha(float4 a, V3 dir) {
  float r = 0.0f;
  if (dir.x != 0.0f) r = __fmul_rn(a.x, fabsf(dir.x));
  if (dir.y != 0.0f) r = __fmaf_rn(a.y, fabsf(dir.y), r);
  if (dir.z != 0.0f) r = __fmaf_rn(dir.z < 0.0f ? a.z : a.w, fabsf(dir.z), r);
  return r;
}

// sum_k a_k * textureLod(map idx_k, u, lod), lod >= 0.  Positions with a
// coordinate of magnitude >= 1e6 (or not finite) sample 0; CHECK = false
// when the caller knows the position is sane.
template <int SAMPLER, bool ISO, int STORAGE, bool CHECK = true, bool FIXED = false>
__device__ __forceinline__ float4 sample_voxel(const MapSet& m, V3 u, int ix, int iy, int iz, V3 ad, float lod) {
  if (SAMPLER == VCT_SAMPLER_EXACT) return sample_exact<ISO, STORAGE>(m, u, ix, iy, iz, ad, lod);
  if (CHECK && !u_sane(u)) return f4(0.f, 0.f, 0.f, 0.f);
  const float wsum = ad.x + ad.y + ad.z;
  if (lod < 1.0f) {
    const float4 t0 = tex3D<float4>(m.l0_tex, u.x, u.y, u.z);
    if (!(lod > 0.0f)) return mul4(t0, wsum);
    float4 t1;
    if (ISO) t1 = tex3DLod<float4>(m.tex[0], u.x, u.y, u.z, 0.0f) * wsum;
    else t1 = aniso_fetch<FIXED>(m, u, ix, iy, iz, ad, 0.0f);
    return fma4(t1, lod, mul4(t0, __fmul_rn(1.0f - lod, wsum)));
  }
  const float l = lod - 1.0f;
  if (ISO) return tex3DLod<float4>(m.tex[0], u.x, u.y, u.z, l) * wsum;
  return aniso_fetch<FIXED>(m, u, ix, iy, iz, ad, l);
}

// The alpha of sample_voxel (texture unit, anisotropic maps) from the alpha
// chains, with the same arithmetic as the alpha channel there.
template <bool FIXED>
__device__ __forceinline__ float sample_alpha(const MapSet& m, V3 u, V3 dir, float lod) {
  float t0 = 0.0f;
  if (lod < 1.0f) t0 = tex3D<float4>(m.l0_tex, u.x, u.y, u.z).w;
  const float t1 = combine_alpha(alpha_fetch<FIXED>(m, u, dir, fmaxf(lod - 1.0f, 0.0f)), dir);
  if (!(lod < 1.0f)) return t1;
  const float wsum = fabsf(dir.x) + fabsf(dir.y) + fabsf(dir.z);
  if (!(lod > 0.0f)) return __fmul_rn(t0, wsum);
  return __fmaf_rn(t1, lod, __fmul_rn(t0, __fmul_rn(1.0f - lod, wsum)));
}

// ------------------------------------------------------------ cone march ----
// Exact early exit: a sample whose position lies more than half the coarsest
// texel outside [0,1] along an axis reads only border texels (0) at every
// level -- a filtered fetch at level l reads texels whose centres lie within
// one texel (2^l / N) of the position, and the coarsest level is L-1.  A cone
// moving away from the volume along an axis is past margin = 3/4 of the
// coarsest texel (MapSet::exit_margin, set by the host) beyond
// `exit_distance`, and adds exact zeros from there on, so its march ends
// there (the extra quarter texel absorbs the rounding of the division).
// Diffuse cones that pass the room's walls (their alpha stays below 1 at the
// coarse levels) otherwise march on to sqrt(3) outside the grid.
__device__ __forceinline__ float exit_distance(const MapSet& m, V3 origin, V3 dir, float max_dist) {
  const float lo = -m.exit_margin, hi = 1.0f + m.exit_margin;
  float d = max_dist;
  if (dir.x > 0.0f) d = fminf(d, (hi - origin.x) / dir.x);
  if (dir.x < 0.0f) d = fminf(d, (lo - origin.x) / dir.x);
  if (dir.y > 0.0f) d = fminf(d, (hi - origin.y) / dir.y);
  if (dir.y < 0.0f) d = fminf(d, (lo - origin.y) / dir.y);
  if (dir.z > 0.0f) d = fminf(d, (hi - origin.z) / dir.z);
  if (dir.z < 0.0f) d = fminf(d, (lo - origin.z) / dir.z);
  return d;  // (+inf margin: max_dist)
}

// Exact empty-space skip: true when every texel the sample at u with this
// lod reads is 0 (MapSet::occ).  Its coarser quadrilinear level is c (level
// 1 when lod < 1, where level 0 and level 1 are read); there the lookup reads
// texels k .. k+1 along each axis, k = floor(u * (N >> c) - 0.5), and the
// finer level's texels lie inside them, so the occ bit of k decides.  Within
// 1/64 texel of a texel boundary the texture unit's fixed-point coordinate
// could pick the neighbouring pair: such samples are fetched.  The test runs
// in 8.8 fixed point: q = floor(256 t) (t scaled by a power of two, so the
// same rounding), k = q >> 8, and the fraction's top byte q & 255 in
// [252, 255] or [0, 3] marks the band (a superset of |frac - 0| < 1/64 and
// frac > 1 - 1/64: conservative).  A pair outside
// the grid is tested at the nearest cell inside it (conservative: border
// texels are 0, and cones leaving the grid stop at exit_distance).  (A position
// that is not finite or is huge ends up clamped or fetched; the texture path
// returns 0 for it either way.)
__device__ __forceinline__ bool sample_empty(const MapSet& m, V3 u, float lod) {
  const int c = min((int)lod + 1, m.L - 1);  // lod >= 0
  const int s = m.N >> c;
  const float fs = (float)(s << 8);
  // (huge or non-finite coordinates saturate or give 0: clamped or fetched)
  const int qx = __float2int_rd(__fmaf_rn(u.x, fs, -128.0f)), qy = __float2int_rd(__fmaf_rn(u.y, fs, -128.0f)),
            qz = __float2int_rd(__fmaf_rn(u.z, fs, -128.0f));
  if ((((uint32_t)qx + 4u) & 255u) < 8u || (((uint32_t)qy + 4u) & 255u) < 8u || (((uint32_t)qz + 4u) & 255u) < 8u)
    return false;
  const int kx = min(max(qx >> 8, 0), s - 1), ky = min(max(qy >> 8, 0), s - 1), kz = min(max(qz >> 8, 0), s - 1);
  const uint32_t w = __ldg(m.occ[c] + ((uint32_t)kz * s + ky) * m.occ_wpr[c] + (kx >> 5));
  return ((w >> (kx & 31)) & 1u) == 0u;
}

#ifndef VCT_SKIP_EMPTY_RGBA
#define VCT_SKIP_EMPTY_RGBA 1
#endif
constexpr bool kSkipEmptyRGBA = VCT_SKIP_EMPTY_RGBA != 0;  // also in the RGBA cones (else shadow cones only)
#ifndef VCT_SKIP_MAX_LOD
#define VCT_SKIP_MAX_LOD 5.0f
#endif
// RGBA cones test for empty space only below this lod: coarser samples are
// fetched without the test (the coarse cells are rarely empty; fetching a
// sample that is empty adds the same exact zeros).  Measured on the 1080p
// bench frame (trace ms): no cap 2.580, below 6 2.552, 5.5 2.550, 5 2.540,
// 4 2.572; the frames are bit-identical.
constexpr float kSkipMaxLod = VCT_SKIP_MAX_LOD;

// The lod of a march step, max(log2(diam * N), 0) with the fast log2
// (lg2.approx).  Its argument is at least 3 * aperture >= 0.05 (the first
// step is at 3 voxels and apertures are >= 0.0174533), never subnormal, so
// the flush-to-zero form gives the same result without the subnormal path.
#ifndef VCT_LOD_FTZ
#define VCT_LOD_FTZ 1
#endif
__device__ __forceinline__ float cone_lod(float x) {
#if VCT_LOD_FTZ
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaxf(r, 0.0f);
#else
  return fmaxf(__log2f(x), 0.0f);
#endif
}

// The sample position origin + dir * dist of a march step, one rounding per
// coordinate (an explicit fused multiply-add, so that it does not depend on
// how the compiler arranges the step loop).
__device__ __forceinline__ V3 march_pos(V3 origin, V3 dir, float dist) {
  return v3(__fmaf_rn(dir.x, dist, origin.x), __fmaf_rn(dir.y, dist, origin.y), __fmaf_rn(dir.z, dist, origin.z));
}

// Whether every position of a march from `origin` along unit `dir` up to
// `stop` is sane (|coordinate| < 1e6, finite); then the step loop needs no
// per-sample check.
__device__ __forceinline__ bool march_sane(V3 origin, V3 dir, float stop) {
  const float reach = fmaxf(fabsf(origin.x), fmaxf(fabsf(origin.y), fabsf(origin.z))) + fmaxf(stop, 0.0f);
  return reach < 1.0e6f && isfinite(dir.x + dir.y + dir.z);
}

#ifndef VCT_TRACE_PIPE
#define VCT_TRACE_PIPE 1
#endif
// Step loop of the texture-unit anisotropic march: 0 = one step after the
// other; 1 = the next step's position, lod and empty-space test (with its
// occupancy load) run while this step's texture fetches are in flight;
// 2 = also the next step's fetches are issued before this step's results
// are used (two sets of results live).  Same samples, same arithmetic.
constexpr int kTracePipe = VCT_TRACE_PIPE;

// The raw texture results of one step of the anisotropic march (the
// fetches of sample_voxel, texture unit, anisotropic maps).
struct Taps {
  float4 t0, x, y, z;
};

template <bool FIXED>
__device__ __forceinline__ void issue_taps(const MapSet& m, V3 u, int oct, V3 ad, float lod, Taps& t) {
  float l = lod - 1.0f;
  if (lod < 1.0f) {
    t.t0 = tex3D<float4>(m.l0_tex, u.x, u.y, u.z);
    if (!(lod > 0.0f)) return;
    l = 0.0f;
  }
  if (ad.x != 0.0f) t.x = axis_fetch<0, FIXED>(m, u, oct & 1, l);
  if (ad.y != 0.0f) t.y = axis_fetch<2, FIXED>(m, u, oct & 2, l);
  if (ad.z != 0.0f) t.z = axis_fetch<4, FIXED>(m, u, oct & 4, l);
}

// sample_voxel<HW, aniso> from the step's taps, operation for operation.
__device__ __forceinline__ float4 combine_taps(const Taps& t, V3 ad, float lod) {
  const float wsum = ad.x + ad.y + ad.z;
  if (lod < 1.0f && !(lod > 0.0f)) return mul4(t.t0, wsum);
  float4 r = f4(0.f, 0.f, 0.f, 0.f);
  if (ad.x != 0.0f) r = mul4(t.x, ad.x);
  if (ad.y != 0.0f) r = fma4(t.y, ad.y, r);
  if (ad.z != 0.0f) r = fma4(t.z, ad.z, r);
  if (lod < 1.0f) return fma4(r, lod, mul4(t.t0, __fmul_rn(1.0f - lod, wsum)));
  return r;
}

// trace_cone for the texture unit and anisotropic maps with the step loop
// software-pipelined (kTracePipe): the march, the samples taken and the
// accumulation are those of the plain loop in trace_cone.
template <bool FIXED>
__device__ float4 trace_cone_pipe(const MapSet& m, V3 origin, V3 dir, float aperture, float max_dist) {
  dir = normalize(dir);
  const int oct = octant(dir);
  const V3 ad = vabs(dir);
  const float cube_res = (float)m.N;
  const float voxel_size = 1.0f / cube_res;
  float4 acc = f4(0.f, 0.f, 0.f, 0.f);
  float dist = 3.0f * voxel_size;
  float diam = dist * aperture;
  V3 sp = march_pos(origin, dir, dist);
  const float stop = exit_distance(m, origin, dir, max_dist);
  const bool check = !march_sane(origin, dir, stop);
  if (!(dist < stop)) return acc;
  float mip = cone_lod(diam * cube_res);
  bool live = !(kSkipEmptyRGBA && m.skip_empty && mip < kSkipMaxLod && sample_empty(m, sp, mip)) && !(check && !u_sane(sp));
  Taps t;
  if (live) issue_taps<FIXED>(m, sp, oct, ad, mip, t);
  while (true) {
    // the next step (taken only while this one leaves alpha below 1)
    const float step = fmaxf(diam * 0.5f, voxel_size);
    dist += step;
    diam = dist * aperture;
    sp = march_pos(origin, dir, dist);
    const bool more = dist < stop;
    const float mip_n = cone_lod(diam * cube_res);
    const bool live_n =
        more && !(kSkipEmptyRGBA && m.skip_empty && mip_n < kSkipMaxLod && sample_empty(m, sp, mip_n)) && !(check && !u_sane(sp));
    if (kTracePipe >= 2) {
      Taps tn;
      if (live_n) issue_taps<FIXED>(m, sp, FIXED ? oct : again(oct), ad, mip_n, tn);
      if (live) acc = fma4(combine_taps(t, ad, mip), 1.0f - acc.w, acc);
      if (!(acc.w < 1.0f) || !more) break;
      t = tn;
    } else {
      if (live) acc = fma4(combine_taps(t, ad, mip), 1.0f - acc.w, acc);
      if (!(acc.w < 1.0f) || !more) break;
      if (live_n) issue_taps<FIXED>(m, sp, FIXED ? oct : again(oct), ad, mip_n, t);
    }
    mip = mip_n;
    live = live_n;
  }
  return acc;
}

// trace_cone, voxel_cone_tracing.frag:88-119.
template <int SAMPLER, bool ISO, int STORAGE, bool FIXED = false>
__device__ float4 trace_cone(const MapSet& m, V3 origin, V3 dir, float aperture, float max_dist) {
  if (kTracePipe > 0 && SAMPLER == VCT_SAMPLER_HW && !ISO) return trace_cone_pipe<FIXED>(m, origin, dir, aperture, max_dist);
  dir = normalize(dir);
  const int ix = dir.x < 0.0f ? 0 : 1, iy = dir.y < 0.0f ? 2 : 3, iz = dir.z < 0.0f ? 4 : 5;
  const V3 ad = vabs(dir);
  const float cube_res = (float)m.N;
  const float voxel_size = 1.0f / cube_res;
  float4 acc = f4(0.f, 0.f, 0.f, 0.f);
  float dist = 3.0f * voxel_size;
  float diam = dist * aperture;
  V3 sp = march_pos(origin, dir, dist);
  const float stop = exit_distance(m, origin, dir, max_dist);
  const bool check = !march_sane(origin, dir, stop);
  while (acc.w < 1.0f && dist < stop) {
    const float mip = cone_lod(diam * cube_res);
    if (!(kSkipEmptyRGBA && m.skip_empty && mip < kSkipMaxLod && sample_empty(m, sp, mip)) && !(check && !u_sane(sp))) {
      // (an empty or insane sample adds exact zeros)
      const float4 s = sample_voxel<SAMPLER, ISO, STORAGE, false>(m, sp, ix, iy, iz, ad, mip);
      acc = fma4(s, 1.0f - acc.w, acc);
    }
    const float step = fmaxf(diam * 0.5f, voxel_size);
    dist += step;
    diam = dist * aperture;
    sp = march_pos(origin, dir, dist);
  }
  return acc;
}

// trace_cone(...).a (trace_shadow, :121-124) with the texture unit over the
// alpha chains: the same march and the same alpha arithmetic, one texture
// fetch per step instead of three.  Every step is sampled (a march
// without empty-space skipping); trace_shadow is the one that skips.
__device__ float trace_alpha(const MapSet& m, V3 origin, V3 dir, float aperture, float max_dist) {
  dir = normalize(dir);
  const float cube_res = (float)m.N;
  const float voxel_size = 1.0f / cube_res;
  float a = 0.0f;
  float dist = 3.0f * voxel_size;
  float diam = dist * aperture;
  const float stop = exit_distance(m, origin, dir, max_dist);
  const bool check = !march_sane(origin, dir, stop);
  while (a < 1.0f && dist < stop) {
    const V3 sp = march_pos(origin, dir, dist);
    if (!(check && !u_sane(sp))) {
      const float lod = cone_lod(diam * cube_res);
      a = __fmaf_rn(sample_alpha<false>(m, sp, dir, lod), 1.0f - a, a);
    }
    dist += fmaxf(diam * 0.5f, voxel_size);
    diam = dist * aperture;
  }
  return a;
}

// ---- shadow cones -----------------------------------------------------------
// A shadow cone is mostly empty space (bench frame: 48 of its 58 steps), so
// what it costs is the loop around the samples.  Its step schedule is the
// same for every pixel, and is read from a table (ShadowGroup) instead of
// being recomputed: recurrence, lg2, level and addressing constants.  Four
// steps go together: one occupancy test at a coarse level whose 3x3x3
// block of cells covers everything the four samples read skips them all;
// else the four steps are tested at the group's own level and the ones that
// are not empty are sampled, in order.  All tests are conservative (below),
// and a sample that is skipped adds exact zeros, so the result is that of the
// full march.  Bench frame: 277 M -> 155 M warp
// instructions (with the pixels' set-up), 290 -> 165 us.
constexpr float kShadowAperture = 0.1f;
#ifndef VCT_SHADOW_UNROLL
#define VCT_SHADOW_UNROLL 1
#endif

// occ3 test of the cell that holds origin + dir * d (see ShadowGroup).  The
// cell is exact up to one rounding of the position; occ3 covers one cell
// each way, and a lookup reads texels within 1.5 of the position.
__device__ __forceinline__ uint32_t shadow_occ(const uint32_t* __restrict__ occ, V3 origin, V3 dir, float d,
                                               float cells, uint32_t base, uint32_t zmul, uint32_t ymul) {
  const float big = 8388608.0f;  // 2^23: floor by the rounding of the sum
  const uint32_t x = __float_as_uint(__fmaf_rd(__saturatef(__fmaf_rn(dir.x, d, origin.x)), cells, big));
  const uint32_t y = __float_as_uint(__fmaf_rd(__saturatef(__fmaf_rn(dir.y, d, origin.y)), cells, big));
  const uint32_t z = __float_as_uint(__fmaf_rd(__saturatef(__fmaf_rn(dir.z, d, origin.z)), cells, big));
  const uint32_t w = __ldg(occ + (z * zmul + (y * ymul + base) + (x >> 5)));
  return (w >> (x & 31u)) & 1u;
}

// The occlusion along `dir` (trace_shadow): ALPHA reads the alpha chains
// (texture unit, anisotropic maps), else the maps; SKIP: empty-space skipping
// is on.
template <int SAMPLER, bool ISO, int STORAGE, bool ALPHA, bool SKIP, bool FIXED = false>
__device__ __forceinline__ float trace_shadow(const MapSet& m, const ShadowGroup* sched, V3 origin, V3 dir,
                                              float max_dist) {
  if constexpr (!SKIP) {
    if constexpr (ALPHA) return trace_alpha(m, origin, dir, kShadowAperture, max_dist);
    else return trace_cone<SAMPLER, ISO, STORAGE>(m, origin, dir, kShadowAperture, max_dist).w;
  }
  dir = normalize(dir);
  const float stop = exit_distance(m, origin, dir, max_dist);
  // (a march with a position that is not sane takes no sample at all: its
  // direction is not finite, and the origin and `stop` are bounded here)
  if (!march_sane(origin, dir, stop)) return 0.0f;
  const int ix = dir.x < 0.0f ? 0 : 1, iy = dir.y < 0.0f ? 2 : 3, iz = dir.z < 0.0f ? 4 : 5;
  const uint32_t* occ = m.occ[1];
  const ShadowGroup* g = sched;
  float a = 0.0f;
  VCT_UNROLL_N(VCT_SHADOW_UNROLL)
  for (float next = 3.0f * (1.0f / (float)m.N); next < stop; ++g) {
    const float4* q = reinterpret_cast<const float4*>(g);
    const float4 q0 = q[0], q1 = q[1];  // (mid, cells, base, zmul), (ymul, next, cells1, base1)
    next = q1.y;
    if (q0.y > 0.0f && !shadow_occ(occ, origin, dir, q0.x, q0.y, __float_as_uint(q0.z), __float_as_uint(q0.w),
                                   __float_as_uint(q1.x)))
      continue;
    const float4 q2 = q[2], qd = q[3];  // (zmul1, ymul1, -, -), dist
    const uint32_t base = __float_as_uint(q1.w), zm = __float_as_uint(q2.x), ym = __float_as_uint(q2.y);
    uint32_t todo = shadow_occ(occ, origin, dir, qd.x, q1.z, base, zm, ym);
    todo |= shadow_occ(occ, origin, dir, qd.y, q1.z, base, zm, ym) << 1;
    todo |= shadow_occ(occ, origin, dir, qd.z, q1.z, base, zm, ym) << 2;
    todo |= shadow_occ(occ, origin, dir, qd.w, q1.z, base, zm, ym) << 3;
    if (!(qd.w < stop)) todo &= (qd.x < stop ? 1u : 0u) | (qd.y < stop ? 2u : 0u) | (qd.z < stop ? 4u : 0u);
#pragma unroll 1
    while (todo) {
      const int i = __ffs(todo) - 1;
      todo &= todo - 1u;
      const float lod = g->lod[i];
      const V3 u = march_pos(origin, dir, g->dist[i]);
      float t;
      if constexpr (ALPHA) t = sample_alpha<FIXED>(m, u, dir, lod);
      else t = sample_voxel<SAMPLER, ISO, STORAGE, false, FIXED>(m, u, ix, iy, iz, vabs(dir), lod).w;
      a = __fmaf_rn(t, 1.0f - a, a);
      if (!(a < 1.0f)) return a;
    }
  }
  return a;
}

// ---- diffuse cones from their schedule ----------------------------------------
// The empty test of sample_empty with the step's constants from its schedule
// entry: t = clamp(coordinate,
// lo, 1) * cells + offset is k * 256 + its fraction, biased by 4 so that the
// band around a texel boundary is one comparison.  The clamp keeps positions
// outside the grid in the nearest cell, out of the band.
__device__ __forceinline__ bool cone_empty(const uint32_t* __restrict__ occ, V3 u, const ConeStep& s) {
  const float off = 8388608.0f - 124.0f;  // 2^23 - 128 + 4
  const uint32_t x = __float_as_uint(__fmaf_rd(fminf(fmaxf(u.x, s.lo), 1.0f), s.cells, off));
  const uint32_t y = __float_as_uint(__fmaf_rd(fminf(fmaxf(u.y, s.lo), 1.0f), s.cells, off));
  const uint32_t z = __float_as_uint(__fmaf_rd(fminf(fmaxf(u.z, s.lo), 1.0f), s.cells, off));
  if (!((x & 0xf8u) && (y & 0xf8u) && (z & 0xf8u))) return false;
  const uint32_t w = __ldg(occ + ((z >> 8) * s.zmul + ((y >> 8) * s.ymul + s.base) + (x >> 13)));
  return ((w >> ((x >> 8) & 31u)) & 1u) == 0u;
}

// Issues the fetches of a sample at lod 1 + l, l >= 0 (issue_taps), and
// sums them (combine_taps).
template <bool ISO, bool FIXED>
__device__ __forceinline__ void far_taps(const MapSet& m, V3 u, int oct, V3 ad, float l, Taps& t) {
  if (ISO) {
    t.x = tex3DLod<float4>(m.tex[0], u.x, u.y, u.z, l);
    return;
  }
  if (ad.x != 0.0f) t.x = axis_fetch<0, FIXED>(m, u, oct & 1, l);
  if (ad.y != 0.0f) t.y = axis_fetch<2, FIXED>(m, u, oct & 2, l);
  if (ad.z != 0.0f) t.z = axis_fetch<4, FIXED>(m, u, oct & 4, l);
}
template <bool ISO>
__device__ __forceinline__ float4 far_combine(const Taps& t, V3 ad) {
  if (ISO) return t.x * (ad.x + ad.y + ad.z);
  float4 r = f4(0.f, 0.f, 0.f, 0.f);
  if (ad.x != 0.0f) r = mul4(t.x, ad.x);
  if (ad.y != 0.0f) r = fma4(t.y, ad.y, r);
  if (ad.z != 0.0f) r = fma4(t.z, ad.z, r);
  return r;
}

// The first sample of a diffuse cone (schedule entry e; unit direction):
// below lod 1 for the nine cones, so it may read level 0 too.
template <bool ISO, bool FIXED = false>
__device__ __forceinline__ float4 cone_first(const MapSet& m, V3 origin, V3 dir, const ConeStep& e) {
  const V3 u = march_pos(origin, dir, e.dist);
  if (m.skip_empty && e.cells > 0.0f && cone_empty(m.occ[1], u, e)) return f4(0.f, 0.f, 0.f, 0.f);
  const int ix = dir.x < 0.0f ? 0 : 1, iy = dir.y < 0.0f ? 2 : 3, iz = dir.z < 0.0f ? 4 : 5;
  const float4 s = sample_voxel<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8, false, FIXED>(m, u, ix, iy, iz, vabs(dir), e.lod);
  return fma4(s, 1.0f, f4(0.f, 0.f, 0.f, 0.f));
}

// tangent, :126-134.
__device__ __forceinline__ V3 tangent(V3 n) {
  const V3 t1 = cross(n, v3(0.f, 0.f, 1.f)), t2 = cross(n, v3(0.f, 1.f, 0.f));
  return length(t1) > length(t2) ? normalize(t1) : normalize(t2);
}
__device__ __forceinline__ V3 mixv(V3 a, V3 b, float t) { return a * (1.0f - t) + b * t; }

// ---- groups that share far fields -------------------------------------------
constexpr float kShareCos = 0.99f;
constexpr float kShareDist = 2.0f;  // voxels
// (A sharing group: kShareW x 2 pixels of a warp's block.)

// Direction (unnormalised) and aperture of diffuse cone k, as trace_diffuse
// computes them from the normal n and its frame o1, o2.
__device__ __forceinline__ V3 diffuse_dir(int cone_set, const ConeRing& ring, V3 n, V3 o1, V3 o2, int k, float& ap) {
  if (cone_set == VCT_CONES_SIX60) {
    ap = kSixAperture;
    const V3 nn = normalize(n);
    if (k == 0) return nn;
    const float sphi = ring.sphi[k - 1], cphi = ring.cphi[k - 1];
    return nn * 0.5f + (o1 * cphi + o2 * sphi) * 0.86602540378f;
  }
  ap = kTan22_5;
  if (k == 0) return n;
  const int j = k - 1;
  // o1, -o1, o2, -o2, c1, -c1, c2, -c2 with c1, c2 = (o1 +- o2) / 2: computed
  // when asked for, so that a loop over the cones does not hold them
  const V3 c = (o1 + o2 * (j < 6 ? 1.0f : -1.0f)) * 0.5f;
  const V3 b = j < 2 ? o1 : (j < 4 ? o2 : c);
  const V3 side = (j & 1) ? -b : b;
  return mixv(n, side, 0.5f);
}

__device__ __forceinline__ V3 refract(V3 I, V3 N, float eta) {
  const float d = dot(N, I);
  const float k = 1.0f - eta * eta * (1.0f - d * d);
  if (k < 0.0f) return v3(0.f, 0.f, 0.f);
  return I * eta - N * (eta * d + sqrtf(k));
}
__device__ __forceinline__ V3 reflect(V3 I, V3 N) { return I - N * (2.0f * dot(N, I)); }

__device__ __forceinline__ V3 mat3v(const float* f) { return v3(f[0], f[1], f[2]); }

// Unit direction to and distance of light i, texture space.
__device__ __forceinline__ void light_dir(const SceneParams& sp, int i, V3 pos, V3& ld, float& d) {
  const vct_point_light& L = sp.lights[i];
  V3 lp = v3(L.position[0] / sp.cube_size, L.position[1] / sp.cube_size, L.position[2] / sp.cube_size);
  lp = lp * 0.5f + v3(0.5f, 0.5f, 0.5f);
  ld = lp - pos;
  d = length(ld);
  ld = normalize(ld);
}

// direct_light, :175-218.
// SPLIT: the shadow cones' occlusion comes from `occlusion` (one value per
// light, `stride` apart), else they are traced here through a batch's maps
// (texture unit, anisotropic RGBA8, alpha chains, empty-space skipping).
template <bool SPLIT>
__device__ V3 direct_light(const SceneParams& sp, const MapSet& m, int enable_shadow, const vct_material_data& mat,
                           V3 pos, V3 nrm, V3 view_dir, const float* occlusion, size_t stride) {
  V3 result = v3(0.f, 0.f, 0.f);
  const int nl = min(sp.n_lights, kMaxLights);
  for (int i = 0; i < nl; ++i) {
    const vct_point_light& L = sp.lights[i];
    V3 ld;
    float d;
    light_dir(sp, i, pos, ld, d);
    const float cs = fmaxf(dot(nrm, ld), 0.0f);
    const V3 lc = v3(L.color[0], L.color[1], L.color[2]) * ((1.0f / (1.0f + d * d)) * cs * L.intensity);
    float shadow = 1.0f;
    if (enable_shadow) {
      float occ;
      if constexpr (SPLIT) occ = occlusion[i * stride];
      else occ = trace_shadow<VCT_SAMPLER_HW, false, VCT_STORAGE_RGBA8, true, true>(m, m.sched->shadow.group, pos, ld, d);
      shadow = fmaxf(0.0f, 1.0f - occ);
    }
    const float lambert = fmaxf(dot(ld, nrm), 0.0f);
    float refract_angle = 0.0f;
    if (mat.dissolve <= 0.1f) {
      const V3 rf = refract(view_dir, nrm, 1.0f / mat.ior);
      refract_angle = fmaxf((1.0f - mat.dissolve) * dot(rf, ld), 0.0f);
    }
    const V3 hv = normalize(ld + view_dir);
    float sa = fmaxf(dot(hv, nrm), 0.0f);
    sa = fmaxf(sa, refract_angle);
    const float sc = powf(sa, mat.shininess);
    const V3 term = mat3v(mat.diffuse) * lambert + mat3v(mat.specular) * sc;
    result = result + mulv(term, lc) * (shadow + 0.04f);
  }
  return result + v3(clamp01(mat.emission[0]), clamp01(mat.emission[1]), clamp01(mat.emission[2]));
}

__device__ __forceinline__ bool refracts(const vct_material_data& mat) {
  return mat.illum == 4 || mat.illum == 6 || mat.illum == 7 || mat.illum == 9;
}

__device__ __forceinline__ float specular_aperture(float shininess) {  // :220-227
  const float r = sqrtf(2.0f / (shininess + 2.0f));
  const float a = tanf(1.57079f * r);
  return fminf(fmaxf(a, 0.0174533f), 3.14159265f);
}

__device__ __forceinline__ unsigned char unorm8(float v) {
  return (unsigned char)__float2uint_rz(clamp01(v) * 255.0f + 0.5f);
}

// The pixel of this lane in a 16-pixel-wide CTA tile at (x0, y0) of the
// shared-far-field kernels: a warp is a kShareWarpW x (32 / kShareWarpW)
// block (lane = x + kShareWarpW y), 16 / kShareWarpW blocks per row of
// blocks.  (One kernel with every phase inside, on the 1920x1080 bench frame,
// trace ms: 16 x 2 strips 1.235, 8 x 4 blocks 1.217, 4 x 8 blocks 1.221.)
__device__ __forceinline__ void share_tile_px(int x0, int y0, int& px, int& py) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  px = x0 + (w % (16 / kShareWarpW)) * kShareWarpW + lane % kShareWarpW;
  py = y0 + (w / (16 / kShareWarpW)) * (32 / kShareWarpW) + lane / kShareWarpW;
}

// Whether this lane's pixel shares the far fields of its group's
// representative (lane `rep`; the lane itself if the group has none).  All
// 32 lanes together; `valid`: the pixel's diffuse cones are traced.
__device__ __forceinline__ bool group_share(int N, bool valid, V3 pos, V3 nrm, int& rep) {
  const int lane = threadIdx.x & 31;
  const unsigned vmask = __ballot_sync(0xffffffffu, valid);
  // this lane's group: columns kShareW * gx .., rows 2 gy and 2 gy + 1 of the block
  const int gx = (lane % kShareWarpW) / kShareW, gy = lane / (2 * kShareWarpW);
  const unsigned grow = ((1u << kShareW) - 1u) << (kShareW * gx);
  const unsigned qv = vmask & ((grow << (2 * kShareWarpW * gy)) | (grow << (2 * kShareWarpW * gy + kShareWarpW)));
  rep = qv ? __ffs(qv) - 1 : lane;
  const V3 rpos = v3(__shfl_sync(0xffffffffu, pos.x, rep), __shfl_sync(0xffffffffu, pos.y, rep),
                     __shfl_sync(0xffffffffu, pos.z, rep));
  const V3 rn = v3(__shfl_sync(0xffffffffu, nrm.x, rep), __shfl_sync(0xffffffffu, nrm.y, rep),
                   __shfl_sync(0xffffffffu, nrm.z, rep));
  bool share = false;
  if (valid) {
    const float lim = kShareDist / (float)N;
    share = dot(normalize(nrm), normalize(rn)) >= kShareCos && fabsf(pos.x - rpos.x) <= lim &&
            fabsf(pos.y - rpos.y) <= lim && fabsf(pos.z - rpos.z) <= lim;
  }
  return share;
}

}  // namespace
}  // namespace vct
