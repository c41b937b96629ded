// k_trace_frame.cu -- the ConeTracer of a frame with the texture-unit
// sampler: voxel_cone_tracing.frag main (:246-275) over the G-buffer in two
// launches.
//
//   k_march -- the cones, apart from the pixels' own arithmetic: the far
//              fields of the pixel groups' diffuse cones (far_share) or every
//              pixel's diffuse cones, the shadow cone of every light, the
//              specular and the refracted cone.  Each goes to a buffer.
//   k_shade -- a thread per pixel: the first samples of the diffuse cones
//              with the far fields behind them, the lights, the sum.
//
// Why two: in one kernel every warp holds the registers of its widest phase
// through all of them, and waits for its slowest lane in each.  Marched as
// separate warps of one launch, a cone keeps 48 registers or fewer (40 warps
// on an SM), and warps that wait for the texture unit (far fields, specular
// cones) share an SM with warps that do arithmetic (shadow cones: mostly
// occupancy tests).  Measured (GB300, bench frame 1920x1080, 256^3, trace
// stage, against one kernel with every phase inside): 1.202 -> 0.872 ms,
// 1.0 G -> 0.58 G warp instructions; 1280x720, 128^3: 0.532 -> 0.373; 512^3
// half-float maps: 2.126 -> 1.235; 256x256, 64^3, isotropic: 0.053 -> 0.034.
// k_march (673 us of it) waits for the texture unit (its pipe 68% busy, issue
// 52%), k_shade (195) is bound by instruction issue (71%).  What passes between
// the two costs 200 MB of DRAM a frame, 30 us at its rate, under kernels that
// use at most an eighth of it.
#include <algorithm>
#include <type_traits>

#include "vct_cone.cuh"

namespace vct {
namespace {

#ifndef VCT_MARCH_MIN_BLOCKS
#define VCT_MARCH_MIN_BLOCKS 10
#endif
#ifndef VCT_MARCH_WARPS
#define VCT_MARCH_WARPS 4
#endif
constexpr int kMarchWarps = VCT_MARCH_WARPS;  // warps of a k_march CTA
#ifndef VCT_SHADE_MIN_BLOCKS
#define VCT_SHADE_MIN_BLOCKS 4
#endif

// The representative of the 4x2-pixel group at (gx, gy): its first pixel,
// row by row, whose diffuse cones are traced.
__device__ __forceinline__ bool group_rep(float cube_size, int W, int H, const float4* __restrict__ gb_pos,
                                          const float4* __restrict__ gb_nrm, int gx, int gy, V3& pos, V3& nrm) {
#pragma unroll 1
  for (int i = 0; i < 2 * kShareW; ++i) {
    const int px = gx * kShareW + i % kShareW, py = gy * 2 + i / kShareW;
    if (px >= W || py >= H) continue;
    const size_t p = (size_t)py * W + px;
    const float4 g1 = gb_nrm[p];
    if (__float_as_uint(g1.w) == 0xffffffffu) continue;
    const float4 g0 = gb_pos[p];
    pos = v3(g0.x / cube_size, g0.y / cube_size, g0.z / cube_size) * 0.5f + v3(0.5f, 0.5f, 0.5f);
    nrm = v3(g1.x, g1.y, g1.z);
    if (fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f) return true;
  }
  return false;
}

__device__ __forceinline__ ConeStep load_step(const ConeStep* e) {  // two 16-byte loads
  const float4 a = reinterpret_cast<const float4*>(e)[0], b = reinterpret_cast<const float4*>(e)[1];
  ConeStep s;
  s.dist = a.x;
  s.lod = a.y;
  s.cells = a.z;
  s.lo = a.w;
  s.base = __float_as_uint(b.x);
  s.zmul = __float_as_uint(b.y);
  s.ymul = __float_as_uint(b.z);
  return s;
}

// trace_cone (texture unit) along unit `dir` from schedule step `e` (the
// second or a later one: lod >= 1) with `acc` behind it: the same samples and
// accumulation, software-pipelined as trace_cone_pipe.
template <bool ISO, bool FIXED>
__device__ __forceinline__ float4 march_sched(const MapSet& m, const ConeStep* e, V3 origin, V3 dir, float4 acc) {
  const float stop = exit_distance(m, origin, dir, kMaxDistance);
  // (a direction that is not finite has no sane position: no sample)
  if (!(e->dist < stop) || !march_sane(origin, dir, stop)) return acc;
  const int oct = octant(dir);
  const V3 ad = vabs(dir);
  const bool skip = m.skip_empty != 0;
  const uint32_t* occ = m.occ[1];
  Taps t;
  bool live = false;
#pragma unroll 1
  while (true) {
    // this step's position and empty-space test run while the last step's fetches are in flight
    const ConeStep s = load_step(e++);
    const V3 u = march_pos(origin, dir, s.dist);
    const bool more = s.dist < stop;
    const bool live_n = more && !(skip && s.cells > 0.0f && cone_empty(occ, u, s));
    if (live) acc = fma4(far_combine<ISO>(t, ad), 1.0f - acc.w, acc);
    if (!(acc.w < 1.0f) || !more) return acc;
    live = live_n;
    if (live) far_taps<ISO, FIXED>(m, u, FIXED ? oct : again(oct), ad, s.lod - 1.0f, t);
  }
}

// What k_march has to do, in warps of a 16x16-pixel tile: `diffuse` warps
// for the diffuse cones, then 8 per light, then 8 for the specular cones
// (a warp takes an 8x4-pixel block).
struct MarchPlan {
  int W, H;
  unsigned tiles_x, tiles;
  unsigned diffuse, lights, specular;  // warps, lights, warps
  unsigned per_tile;                   // warps of a tile
  int cone_set;
};

static_assert(trace_far_slots(16, 16) == 32 * 9, "march_far: a lane for each group of a tile");

// The far field of one cone of a tile's 32 groups: lane = group, marched in
// lockstep, so that the lanes read neighbouring texels of the same maps at
// the same step of the schedule.
template <bool ISO>
__device__ __forceinline__ void march_far(float cube_size, const MapSet& m, const MarchPlan& mp, int tx, int ty, int k,
                                          const float4* __restrict__ gb_pos, const float4* __restrict__ gb_nrm,
                                          float4* __restrict__ far, const ConeSchedule& sched, const ConeRing& ring) {
  const int lane = threadIdx.x & 31;
  const int gx = tx * (16 / kShareW) + lane % (16 / kShareW), gy = ty * 8 + lane / (16 / kShareW);
  const int groups_x = (mp.W + kShareW - 1) / kShareW;
  if (gx >= groups_x || gy >= (mp.H + 1) / 2) return;
  V3 origin, n;
  if (!group_rep(cube_size, mp.W, mp.H, gb_pos, gb_nrm, gx, gy, origin, n)) return;
  const V3 o1 = normalize(tangent(n));
  const V3 o2 = normalize(cross(o1, n));
  float ap;
  const V3 dir = normalize(diffuse_dir(mp.cone_set, ring, n, o1, o2, k, ap));
  const int K = mp.cone_set == VCT_CONES_SIX60 ? 6 : 9;
  far[((size_t)gy * groups_x + gx) * K + k] =
      march_sched<ISO, true>(m, sched.step + 1, origin, dir, f4(0.f, 0.f, 0.f, 0.f));
}

// One whole diffuse cone: its first sample, then the march behind it.
// FIXED as in axis_fetch: a frame of whole cones is bound by the filter
// wavefronts alone and marches faster with looked-up handles (per-pixel
// cones, trace 2.62 against 2.69 ms), one with far fields with fixed ones
// (0.872 against 0.918 ms), where the look-ups' registers cost more.
template <bool ISO, bool FIXED>
__device__ __forceinline__ float4 march_cone(const MapSet& m, V3 pos, V3 dir, const ConeSchedule& sched) {
  const float stop = exit_distance(m, pos, dir, kMaxDistance);
  float4 c = f4(0.f, 0.f, 0.f, 0.f);
  if (!(sched.step[0].dist < stop) || !march_sane(pos, dir, stop)) return c;
  c = cone_first<ISO, true>(m, pos, dir, sched.step[0]);
  if (c.w < 1.0f) c = march_sched<ISO, FIXED>(m, sched.step + 1, pos, dir, c);
  return c;
}

// trace_diffuse (:140-168) of a warp's pixels that do not share far fields
// (0.4% of the bench frame's): three pixels (nine cones) or five (six cones)
// at a time, a lane per cone, the cones added up in order.
template <bool ISO>
__device__ __forceinline__ void march_alone(const MapSet& m, int cone_set, unsigned lone, V3 pos, V3 nrm, size_t p,
                                            float4* __restrict__ diffuse, const ConeSchedule& sched,
                                            const ConeRing& ring) {
  const int lane = threadIdx.x & 31;
  const int K = cone_set == VCT_CONES_SIX60 ? 6 : 9, per = 32 / K;
  const int j = lane / K, k = lane - j * K;
  while (lone) {  // warp-uniform
    // the lane's pixel: the j-th of those left
    unsigned mask = lone;
    for (int i = 0; i < j; ++i) mask &= mask - 1u;
    const bool own = j < per && mask;
    const int src = mask ? __ffs(mask) - 1 : 0;
    const V3 o = v3(__shfl_sync(0xffffffffu, pos.x, src), __shfl_sync(0xffffffffu, pos.y, src),
                    __shfl_sync(0xffffffffu, pos.z, src));
    const V3 n = v3(__shfl_sync(0xffffffffu, nrm.x, src), __shfl_sync(0xffffffffu, nrm.y, src),
                    __shfl_sync(0xffffffffu, nrm.z, src));
    const size_t px = __shfl_sync(0xffffffffu, (unsigned long long)p, src);
    float4 c = f4(0.f, 0.f, 0.f, 0.f);
    if (own) {
      const V3 o1 = normalize(tangent(n));
      const V3 o2 = normalize(cross(o1, n));
      float ap;
      c = march_cone<ISO, true>(m, o, normalize(diffuse_dir(cone_set, ring, n, o1, o2, k, ap)), sched);
    }
    V3 acc = v3(0.f, 0.f, 0.f);
    for (int q = 0; q < K; ++q) {
      const int from = min(j * K + q, 31);
      acc = acc + v3(__shfl_sync(0xffffffffu, c.x, from), __shfl_sync(0xffffffffu, c.y, from),
                     __shfl_sync(0xffffffffu, c.z, from));
    }
    acc = acc * (1.0f / (float)K);
    if (own && k == 0) diffuse[px] = f4(acc.x, acc.y, acc.z, 0.f);
    for (int i = 0; i < per && lone; ++i) lone &= lone - 1u;
  }
}

// SHARE: the diffuse warps of a tile are one per cone for the groups' far
// fields, then eight for the pixels that do not share; else eight, each
// marching every cone of its pixels.  ALPHA: the shadow cones read the alpha
// chains; SKIP: empty-space skipping is on.
template <bool ISO, bool SHARE, bool ALPHA, bool SKIP>
__global__ void __launch_bounds__(kMarchWarps * 32, VCT_MARCH_MIN_BLOCKS)
    k_march(SceneParams sp, V3 cam, const __grid_constant__ MapSet m, MarchPlan mp, const float4* __restrict__ gb_pos,
            const float4* __restrict__ gb_nrm, TraceWork tw, const __grid_constant__ ShadowSchedule shadow_sched,
            const __grid_constant__ ConeSchedule sched, const __grid_constant__ ConeRing ring) {
  const unsigned unit = blockIdx.x * kMarchWarps + (threadIdx.x >> 5);
  const unsigned tile = unit / mp.per_tile;
  unsigned r = unit - tile * mp.per_tile;  // the warp's work in its tile
  if (tile >= mp.tiles) return;
  const int tx = (int)(tile % mp.tiles_x), ty = (int)(tile / mp.tiles_x);
  const int lane = threadIdx.x & 31;
  const int K = mp.cone_set == VCT_CONES_SIX60 ? 6 : 9;
  if (SHARE && r < (unsigned)K) {
    march_far<ISO>(sp.cube_size, m, mp, tx, ty, (int)r, gb_pos, gb_nrm, tw.far, sched, ring);
    return;
  }
  if (SHARE) r -= (unsigned)K;
  const int w = (int)(r & 7u);
  static_assert(kShareWarpW == 8, "group_share's lanes are these pixels");
  const int px = tx * 16 + (w & 1) * 8 + (lane & 7), py = ty * 16 + (w >> 1) * 4 + (lane >> 3);
  const size_t p = (size_t)py * mp.W + px;
  bool valid = false;
  V3 pos = v3(0.f, 0.f, 0.f), nrm = v3(0.f, 0.f, 1.f);
  if (px < mp.W && py < mp.H) {
    const float4 g1 = gb_nrm[p];
    if (__float_as_uint(g1.w) != 0xffffffffu) {
      const float4 g0 = gb_pos[p];
      pos = v3(g0.x / sp.cube_size, g0.y / sp.cube_size, g0.z / sp.cube_size) * 0.5f + v3(0.5f, 0.5f, 0.5f);
      nrm = v3(g1.x, g1.y, g1.z);
      valid = fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f;  // within_cube, :250
    }
  }
  const unsigned n_diffuse = mp.diffuse - (SHARE ? (unsigned)K : 0u);
  if (r < n_diffuse) {
    if constexpr (SHARE) {
      int rep;
      const bool share = group_share(m.N, valid, pos, nrm, rep);
      const unsigned lone = __ballot_sync(0xffffffffu, valid && !share);
      if (lone) march_alone<ISO>(m, mp.cone_set, lone, pos, nrm, p, tw.diffuse, sched, ring);
    } else if (valid) {
      V3 acc = v3(0.f, 0.f, 0.f);
#pragma unroll 1
      for (int k = 0; k < K; ++k) {
        // (the tangent frame again for every cone: cheaper than holding it across the march)
        const V3 o1 = normalize(tangent(nrm));
        const V3 o2 = normalize(cross(o1, nrm));
        float ap;
        const float4 c =
            march_cone<ISO, false>(m, pos, normalize(diffuse_dir(mp.cone_set, ring, nrm, o1, o2, k, ap)), sched);
        acc = acc + v3(c.x, c.y, c.z);
      }
      acc = acc * (1.0f / (float)K);
      tw.diffuse[p] = f4(acc.x, acc.y, acc.z, 0.f);
    }
    return;
  }
  if (!valid) return;
  r -= n_diffuse;
  const unsigned light = r >> 3;
  if (light < mp.lights) {
    V3 ld;
    float d;
    light_dir(sp, (int)light, pos, ld, d);
    tw.shadow[(size_t)light * mp.W * mp.H + p] =
        trace_shadow<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8, ALPHA, SKIP, true>(m, shadow_sched.group, pos, ld, d);
    return;
  }
  // the specular cone, and the refracted one of transparent materials
  // (:258-272)
  const float4 g0 = gb_pos[p];
  const vct_material_data& mat = sp.materials[__float_as_uint(g0.w)];
  const V3 view_dir = normalize(v3(g0.x, g0.y, g0.z) - cam);
  const float sap = specular_aperture(mat.shininess);
  const bool through = refracts(mat);
#pragma unroll 1
  for (int pass = 0; pass < (through ? 2 : 1); ++pass) {
    const V3 d = pass == 0 ? normalize(reflect(-view_dir, nrm)) : refract(view_dir, nrm, 1.0f / mat.ior);
    (pass == 0 ? tw.specular : tw.refracted)[p] =
        trace_cone<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8, true>(m, pos, d, sap, kMaxDistance);
  }
}

// The diffuse term of a pixel that shares (far: its group's far fields): each
// cone takes its first sample itself and the far field behind it.  The loop
// is software-pipelined: the next cone's direction, position and empty-space
// test (with its occupancy load) run while this cone's fetches are in flight.
template <bool ISO>
__device__ __forceinline__ V3 shared_diffuse(const MapSet& m, int cone_set, V3 pos, V3 n,
                                             const float4* far, const ConeStep& first,
                                             const ConeRing& ring) {
  const int K = cone_set == VCT_CONES_SIX60 ? 6 : 9;
  const V3 o1 = normalize(tangent(n));
  const V3 o2 = normalize(cross(o1, n));
  const bool skip = m.skip_empty != 0 && first.cells > 0.0f;
  const bool near = first.lod < 1.0f;  // (uniform) the sample reads level 0 too
  const uint32_t* occ = m.occ[1];
  V3 acc = v3(0.f, 0.f, 0.f), dir = v3(0.f, 0.f, 1.f);
  Taps t;
  float4 fk = f4(0.f, 0.f, 0.f, 0.f);
  bool live = false;
#pragma unroll 1
  for (int k = 0; k <= K; ++k) {
    // (the origin is a surface point inside the grid and the first step
    // three voxels: the sample position is sane, and one beyond the grid's
    // exit margin reads border texels, 0, as the unshortened march would)
    float ap;
    V3 dir_n = dir, u = pos;
    bool live_n = false;
    if (k < K) {
      dir_n = normalize(diffuse_dir(cone_set, ring, n, o1, o2, k, ap));
      u = march_pos(pos, dir_n, first.dist);
      live_n = !(skip && cone_empty(occ, u, first));
    }
    if (k > 0) {
      float4 c = f4(0.f, 0.f, 0.f, 0.f);
      if (live) {
        const V3 ad = vabs(dir);
        const float4 s = far_combine<ISO>(t, ad);
        if (near) {
          const float wsum = ad.x + ad.y + ad.z;
          c = first.lod > 0.0f ? fma4(s, first.lod, mul4(t.t0, __fmul_rn(1.0f - first.lod, wsum))) : mul4(t.t0, wsum);
        } else {
          c = s;
        }
      }
      if (c.w < 1.0f) c = fma4(fk, 1.0f - c.w, c);
      acc = acc + v3(c.x, c.y, c.z);
    }
    if (k < K) {
      fk = far[k];
      dir = dir_n;
      live = live_n;
      if (live) {
        if (near) t.t0 = tex3D<float4>(m.l0_tex, u.x, u.y, u.z);
        far_taps<ISO, true>(m, u, octant(dir), vabs(dir), fmaxf(first.lod - 1.0f, 0.0f), t);
      }
    }
  }
  return acc * (1.0f / (float)K);
}

// Shades the pixels (main, voxel_cone_tracing.frag:246-275) from k_march's
// buffers; SHARE: the diffuse term of the pixels that share is taken from
// their group's far fields here, the others' and, without SHARE, every
// pixel's comes from `diffuse` (null: no diffuse term).
template <bool ISO, bool SHARE>
__global__ void __launch_bounds__(256, SHARE ? VCT_SHADE_MIN_BLOCKS : 6)
    k_shade(SceneParams sp, CameraParams cp, const __grid_constant__ MapSet m, TraceParams tp,
            const float4* __restrict__ gb_pos, const float4* __restrict__ gb_nrm, uchar4* __restrict__ frame,
            float4* __restrict__ frame_f32, TraceWork tw, const float4* diffuse,
            const __grid_constant__ ConeStep first, const __grid_constant__ ConeRing ring) {
  follows_previous();  // (the maps it samples were whole before k_march)
  int px, py;
  share_tile_px(blockIdx.x * 16, blockIdx.y * 16, px, py);
  const size_t p = (size_t)py * cp.W + px;
  const bool inside = px < cp.W && py < cp.H;
  bool valid = false;
  V3 pos = v3(0.f, 0.f, 0.f), nrm = v3(0.f, 0.f, 1.f);
  if (inside) {
    const float4 g1 = gb_nrm[p];
    if (__float_as_uint(g1.w) != 0xffffffffu) {
      const float4 g0 = gb_pos[p];
      pos = v3(g0.x / sp.cube_size, g0.y / sp.cube_size, g0.z / sp.cube_size) * 0.5f + v3(0.5f, 0.5f, 0.5f);
      nrm = v3(g1.x, g1.y, g1.z);
      // within_cube(pos, 0) (:61-64, 250): a fragment outside returns without
      // writing; the pixel keeps the clear colour.
      valid = fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f;
    }
  }
  bool share = false;
  if constexpr (SHARE) {
    int rep;
    share = group_share(m.N, valid, pos, nrm, rep);
  }
  if (!inside) return;
  float4 out = f4(0.15f, 0.25f, 0.25f, 1.0f);  // glClearColor, renderer.cpp:398
  if (valid) {
    V3 fd = v3(0.f, 0.f, 0.f), fdir = v3(0.f, 0.f, 0.f), fs = v3(0.f, 0.f, 0.f);
    if (share) {
      const int K = tp.cone_set == VCT_CONES_SIX60 ? 6 : 9;
      const size_t group = (size_t)(py >> 1) * ((cp.W + kShareW - 1) / kShareW) + px / kShareW;
      fd = shared_diffuse<ISO>(m, tp.cone_set, pos, nrm, tw.far + group * K, first, ring);
    } else if (diffuse) {
      const float4 d = diffuse[p];
      fd = v3(d.x, d.y, d.z);
    }
    const float4 g0 = gb_pos[p];
    const vct_material_data& mat = sp.materials[__float_as_uint(g0.w)];
    if (tp.enable_diffuse) fd = mulv(mat3v(mat.diffuse), fd);
    const V3 view_dir = normalize(v3(g0.x, g0.y, g0.z) - v3(cp.cam_pos[0], cp.cam_pos[1], cp.cam_pos[2]));
    if (tp.enable_direct)
      fdir = direct_light<true>(sp, m, tp.enable_shadow, mat, pos, nrm, view_dir, tw.shadow + p,
                                (size_t)cp.W * cp.H);
    if (tp.enable_specular) {
      const float4 c = tw.specular[p];
      fs = mulv(mat3v(mat.specular), v3(c.x, c.y, c.z));
    }
    V3 f = fs + fd + fdir;
    if (refracts(mat) && tp.enable_specular) {
      const float4 c = tw.refracted[p];
      const V3 tr = mulv(mat3v(mat.transmittance), v3(c.x, c.y, c.z));
      f = tr * (1.0f - mat.dissolve) + f * mat.dissolve;
    }
    out = f4(f.x, f.y, f.z, 1.0f);
  }
  frame[p] = make_uchar4(unorm8(out.x), unorm8(out.y), unorm8(out.z), unorm8(out.w));
  if (frame_f32) frame_f32[p] = out;
}

// Builds the schedules (a warp, one thread per schedule: the recurrences are
// serial, and run once per map set).
__global__ void k_cone_schedules(MapSet m, ConeSchedules* __restrict__ out) {
  const float cube_res = (float)m.N;
  const float voxel_size = 1.0f / cube_res;
  float dist = 3.0f * voxel_size;
  if (threadIdx.x == 0) {
    auto level = [&](int c, float& cells, uint32_t& base, uint32_t& zmul, uint32_t& ymul) {
      const int s = m.N >> c;
      cells = __uint_as_float(__float_as_uint((float)s) - 1u);  // so that a coordinate of 1 is in the last cell
      ymul = (uint32_t)m.occ_wpr[c];
      zmul = (uint32_t)s * ymul;
      const uint32_t e = 0x4b000000u;  // the bits of 2^23
      base = (uint32_t)(m.occ3[c] - m.occ[1]) - e * zmul - e * ymul - (e >> 5);
    };
    for (int g = 0; g < kShadowGroups; ++g) {
      ShadowGroup r;
      int c = 1;
      for (int i = 0; i < 4; ++i) {
        const float diam = dist * kShadowAperture;
        r.dist[i] = dist;
        r.lod[i] = cone_lod(diam * cube_res);
        c = max(c, min((int)r.lod[i] + 1, m.L - 1));
        dist += fmaxf(diam * 0.5f, voxel_size);
      }
      r.next = g + 1 < kShadowGroups ? dist : __int_as_float(0x7f800000);
      level(c, r.cells1, r.base1, r.zmul1, r.ymul1);
      // The four-step test's level: the first whose cell is at least as wide
      // as the group's half span plus the reach of its samples, which read
      // texels within 1.5 cells of level c of their positions (a quarter
      // more for rounding).
      const float need = 0.5f * (r.dist[3] - r.dist[0]) * cube_res + 1.75f * (float)(1 << c);
      int t = c;
      while (t < m.L && (float)(1 << t) * 0.97f < need) ++t;
      r.mid = 0.5f * (r.dist[0] + r.dist[3]);
      r.cells = 0.0f;
      r.base = r.zmul = r.ymul = 0u;
      if (t < m.L) level(t, r.cells, r.base, r.zmul, r.ymul);
      r.pad[0] = r.pad[1] = 0.0f;
      out->shadow.group[g] = r;
    }
  } else if (threadIdx.x < 3) {
    const int set = (int)threadIdx.x - 1;
    const float ap = set == VCT_CONES_SIX60 ? kSixAperture : kTan22_5;
    for (int i = 0; i < kConeSteps; ++i) {
      const float diam = dist * ap;
      ConeStep r;
      r.dist = i + 1 < kConeSteps ? dist : __int_as_float(0x7f800000);
      r.lod = cone_lod(diam * cube_res);
      const int c = min((int)r.lod + 1, m.L - 1), s = m.N >> c;
      r.cells = kSkipEmptyRGBA && r.lod < kSkipMaxLod ? (float)(s << 8) : 0.0f;
      r.lo = (0.5f + 8.0f / 256.0f) / (float)s;
      r.ymul = (uint32_t)m.occ_wpr[c];
      r.zmul = (uint32_t)s * r.ymul;
      const uint32_t e = 0x4b000000u;
      r.base = (uint32_t)(m.occ[c] - m.occ[1]) - (e >> 8) * r.zmul - (e >> 8) * r.ymul - (e >> 13);
      r.pad = 0.0f;
      out->cone[set].step[i] = r;
      dist += fmaxf(diam * 0.5f, voxel_size);
    }
  } else if (threadIdx.x < 8) {
    const int k = (int)threadIdx.x - 3;
    sincosf(6.28318530717958648f * (float)k / 5.0f, &out->ring.sphi[k], &out->ring.cphi[k]);
  }
}

template <bool ISO>
cudaError_t run_frame(const SceneParams& sp, const CameraParams& cp, const MapSet& ms, const TraceParams& tp,
                      const float4* gb_pos, const float4* gb_nrm, uchar4* frame, float4* frame_f32,
                      const ConeSchedules& sched, const TraceWork& tw, cudaStream_t st, int* launches) {
  const bool six = tp.cone_set == VCT_CONES_SIX60;
  const bool cones = tp.enable_diffuse && !tp.diffuse_in, share = cones && tp.far_share;
  const ConeSchedule& cone = sched.cone[six ? 1 : 0];
  MarchPlan mp;
  mp.W = cp.W;
  mp.H = cp.H;
  mp.tiles_x = (unsigned)((cp.W + 15) / 16);
  mp.tiles = mp.tiles_x * (unsigned)((cp.H + 15) / 16);
  mp.diffuse = share ? (six ? 6u : 9u) + 8u : (cones ? 8u : 0u);
  mp.lights = tp.enable_direct && tp.enable_shadow ? (unsigned)std::min(std::max(sp.n_lights, 0), kMaxLights) : 0u;
  mp.specular = tp.enable_specular ? 8u : 0u;
  mp.per_tile = mp.diffuse + 8u * mp.lights + mp.specular;
  mp.cone_set = tp.cone_set;
  if (mp.per_tile) {
    const bool skip = ms.skip_empty != 0, alpha = ms.alpha_tex[0] != 0;
    const unsigned long long warps = (unsigned long long)mp.tiles * mp.per_tile;
    const unsigned grid = (unsigned)((warps + kMarchWarps - 1) / kMarchWarps);
    const V3 cam = {cp.cam_pos[0], cp.cam_pos[1], cp.cam_pos[2]};
    auto pick = [&](auto share_tag) {
      constexpr bool S = decltype(share_tag)::value;
      if (ISO || !alpha) return skip ? k_march<ISO, S, false, true> : k_march<ISO, S, false, false>;
      return skip ? k_march<ISO, S, !ISO, true> : k_march<ISO, S, !ISO, false>;
    };
    auto kern = share ? pick(std::true_type()) : pick(std::false_type());
    kern<<<grid, kMarchWarps * 32, 0, st>>>(sp, cam, ms, mp, gb_pos, gb_nrm, tw, sched.shadow, cone, sched.ring);
    if (launches) ++*launches;
  }
  const float4* diffuse = !tp.enable_diffuse ? nullptr : (tp.diffuse_in ? tp.diffuse_in : tw.diffuse);
  const dim3 grid((cp.W + 15) / 16, (cp.H + 15) / 16);
  auto shade = share ? k_shade<ISO, true> : k_shade<ISO, false>;
  cudaError_t e = cudaSuccess;
  if (mp.per_tile)
    e = launch_next(shade, grid, 256, st, sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, tw, diffuse, cone.step[0],
                    sched.ring);
  else
    shade<<<grid, 256, 0, st>>>(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, tw, diffuse, cone.step[0], sched.ring);
  if (launches) ++*launches;
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

cudaError_t launch_cone_schedules(const MapSet& ms, ConeSchedules* out, cudaStream_t st) {
  k_cone_schedules<<<1, 32, 0, st>>>(ms, out);
  return cudaGetLastError();
}

cudaError_t launch_trace(const SceneParams& sp, const CameraParams& cp, const MapSet& ms, const TraceParams& tp,
                         const float4* gb_pos, const float4* gb_nrm, uchar4* frame, float4* frame_f32,
                         const ConeSchedules& sched, const TraceWork& tw, cudaStream_t st, int* launches) {
  if (tp.sampler == VCT_SAMPLER_EXACT || tp.view_voxel_dir < 7)
    return launch_trace_px(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, st, launches);
  if (tp.mip_mode == VCT_MIP_ISO)
    return run_frame<true>(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, sched, tw, st, launches);
  return run_frame<false>(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, sched, tw, st, launches);
}

}  // namespace vct
