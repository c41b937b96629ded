// k_trace.cu -- the ConeTracer in one kernel (voxel_cone_tracing.frag main,
// :246-275, over the G-buffer): the FP32 software sampler (k_trace_exact), the
// voxel debug view (k_view) and a batch's one-launch traces (k_trace_batch*);
// also the learned term's training targets and judge.  A frame with the
// texture-unit sampler is traced by k_trace_frame.cu.
//
// A batch's one-launch trace takes a thread per pixel, in 16x16-pixel tiles of
// 8x4 warp blocks where far fields are shared, so that neighbouring lanes
// march neighbouring, nearly parallel cones and hit the same texture-cache
// lines.
#include <algorithm>

#include "vct_cone.cuh"

namespace vct {
namespace {

#ifndef VCT_TRACE_BATCH_MIN_BLOCKS
#define VCT_TRACE_BATCH_MIN_BLOCKS 3
#endif
// The batched trace keeps a scene's descriptor in shared memory and its
// values in registers, so it is compiled for its own occupancy.
constexpr int kTraceBatchMinBlocks = VCT_TRACE_BATCH_MIN_BLOCKS;

// trace_diffuse, :140-168 (9 equal-weight cones), texture unit; cone set SIX60 (no
// reference counterpart): the normal plus 5 cones 60 degrees off it in the
// same tangent frame, aperture 2 tan(30 deg), equal weights.
template <bool ISO>
__device__ V3 trace_diffuse(const MapSet& m, int cone_set, V3 origin, V3 n) {
  const V3 o1 = normalize(tangent(n));
  const V3 o2 = normalize(cross(o1, n));
  float4 acc = f4(0.f, 0.f, 0.f, 0.f);
  if (cone_set == VCT_CONES_SIX60) {
    const float ap = kSixAperture;
    const V3 nn = normalize(n);
    acc = trace_cone<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8>(m, origin, nn, ap, kMaxDistance);
#pragma unroll 1
    for (int k = 0; k < 5; ++k) {
      const float sphi = m.sched->ring.sphi[k], cphi = m.sched->ring.cphi[k];
      const V3 d = nn * 0.5f + (o1 * cphi + o2 * sphi) * 0.86602540378f;
      acc = acc + trace_cone<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8>(m, origin, d, ap, kMaxDistance);
    }
    return v3(acc.x, acc.y, acc.z) * (1.0f / 6.0f);
  }
  const V3 c1 = (o1 + o2) * 0.5f, c2 = (o1 - o2) * 0.5f;
  acc = trace_cone<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8>(m, origin, n, kTan22_5, kMaxDistance);
  // Side cones o1, -o1, o2, -o2, c1, -c1, c2, -c2 (:156-165), selected
  // arithmetically so that no local-memory array is needed.
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    const V3 b = k < 2 ? o1 : (k < 4 ? o2 : (k < 6 ? c1 : c2));
    const V3 side = (k & 1) ? -b : b;
    acc = acc + trace_cone<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8>(m, origin, mixv(n, side, 0.5f), kTan22_5, kMaxDistance);
  }
  return v3(acc.x, acc.y, acc.z) * (1.0f / 9.0f);
}

// ------------------------------------------------- shared far fields ------
// Far-field sharing (TraceParams::far_share, texture-unit sampler).  The
// diffuse cones of neighbouring pixels on one surface start a fraction of a
// voxel apart in nearly the same directions, and after their first sample
// (3 voxels out, lod log2(3 aperture)) their samples are coarse texels whose
// filtered values barely differ across a few pixels.  So every diffuse cone
// is split after its first step: each pixel takes that sample itself, and the
// rest of the march (the "far field") is done once per group of kShareW x 2
// pixels, along the cones of one pixel of the group (its representative),
// by the lanes of the warp together (far_fields below).  The split is exact
// front-to-back compositing: a march that continues from the first sample s
// equals s + (1 - s.a) * far, where far is the march of the remaining steps
// from zero, and both stop at the same step (alpha reaching 1).  Only the
// representative's positions and directions stand in for the other
// pixels'.  A pixel shares only when its normal is within kShareCos of the
// representative's and its surface point within kShareDist voxels along
// every axis; others march their own cones.  Measured against the FP64
// oracle on the 1080p bench frame (sharing alone, the texture unit's 8-bit
// filter weights being 71 dB): 2x2 groups 80.6 dB, 4x2 groups 73.1 dB, with
// the diffuse cones' two-level texture fetches cut from 238 to 60 and 31
// per pixel.
#ifndef VCT_FIRST_UNROLL
#define VCT_FIRST_UNROLL 1  // the per-pixel first samples of the diffuse cones: cones in flight together
#endif
constexpr int kShareQuads = 16 / kShareW;  // groups of a warp
constexpr int kShareCones = 9;
constexpr int kShareJobs = kShareQuads * kShareCones;

// Order of a warp's far-field jobs: 1 = the jobs that start after the
// first 32 (the last lanes to finish wait for them) are those with the
// shortest exit distance, so the warp's tail is short; 0 = cone-major order.
#ifndef VCT_FAR_SHORT_TAIL
#define VCT_FAR_SHORT_TAIL 1
#endif
constexpr bool kFarShortTail = VCT_FAR_SHORT_TAIL != 0;

struct FarWarp {
  float4 far[kShareJobs];   // far field of cone k of group slot q at q * K + k
  float4 job[kShareJobs];   // job j = k * nq + q: unit direction, exit distance
  float origin[kShareQuads][3];  // representative's texture-space position
  float normal[kShareQuads][3];  // and normal
  uint8_t order[kShareJobs];     // the job handed out n-th
};

// The far fields of a warp's nq groups.  Job j = k * nq + q is cone k of group
// slot q (neighbouring lanes start on the same cone of neighbouring groups,
// which read neighbouring texels).  The lanes first set up every job's
// direction and exit distance together (fw.job), then march: a lane whose
// cone ends (alpha 1, the grid's edge) takes the next job while the others
// march on.  The march starts at the second step of the schedule (dist1,
// diam1) with nothing accumulated.  Results go to fw.far[q * K + k].
__device__ void far_fields(const MapSet& m, FarWarp& fw, int cone_set, int nq, float dist1, float diam1) {
  const int lane = threadIdx.x & 31;
  const int K = cone_set == VCT_CONES_SIX60 ? 6 : 9;
  const int n_jobs = nq * K;
  for (int j = lane; j < n_jobs; j += 32) {
    const int k = j / nq, q = j - k * nq;
    const V3 n = v3(fw.normal[q][0], fw.normal[q][1], fw.normal[q][2]);
    const V3 o1 = normalize(tangent(n));
    const V3 o2 = normalize(cross(o1, n));
    float ap;
    const V3 d = normalize(diffuse_dir(cone_set, m.sched->ring, n, o1, o2, k, ap));
    const V3 o = v3(fw.origin[q][0], fw.origin[q][1], fw.origin[q][2]);
    fw.job[j] = f4(d.x, d.y, d.z, exit_distance(m, o, d, kMaxDistance));
  }
  __syncwarp();
  {
    // Jobs 0..31 start together; the n_jobs - 32 handed out after them
    // (kShareJobs - 32 at most) are swapped for the jobs of shortest exit
    // distance -- the cones that reach least far, nearly always the shortest
    // marches -- picked by warp min-reductions of (distance, job) keys.
    // Which lane marches a job changes nothing in its result.
    static_assert(kShareJobs <= 64, "job index in 6 bits");
    const int n_tail = n_jobs - 32;
    uint64_t tail = 0;  // warp-uniform: the jobs chosen for the tail
    if (kFarShortTail && n_tail > 0) {
      auto key = [&](int j) {
        return j < n_jobs ? (__float_as_uint(fmaxf(fw.job[j].w, 0.0f)) & ~63u) | (unsigned)j : ~0u;
      };
      unsigned k0 = key(lane), k1 = key(lane + 32);
      for (int t = 0; t < n_tail; ++t) {
        const unsigned mn = __reduce_min_sync(0xffffffffu, min(k0, k1));
        tail |= 1ull << (mn & 63u);
        if (k0 == mn) k0 = ~0u;
        if (k1 == mn) k1 = ~0u;
      }
    }
    // chosen jobs among 0..31 trade places, in order, with the jobs at 32..
    // that were not chosen
    // (no choice made: a = b = 0, every job keeps its place)
    const uint32_t a = (uint32_t)tail;
    const uint32_t b = tail ? ~(uint32_t)(tail >> 32) & ((1u << n_tail) - 1u) : 0u;
    auto nth = [](uint32_t mask, int i) {  // the i-th set bit of mask
      for (; i > 0; --i) mask &= mask - 1u;
      return __ffs(mask) - 1;
    };
    for (int j = lane; j < n_jobs; j += 32) {
      int o = j;
      if (j < 32 && ((a >> j) & 1u)) o = 32 + nth(b, __popc(a & ((1u << j) - 1u)));
      if (j >= 32 && ((b >> (j - 32)) & 1u)) o = nth(a, __popc(b & ((1u << (j - 32)) - 1u)));
      fw.order[j] = (uint8_t)o;
    }
  }
  __syncwarp();
  const float ap = cone_set == VCT_CONES_SIX60 ? kSixAperture : kTan22_5;
  const float cube_res = (float)m.N;
  const float voxel_size = 1.0f / cube_res;
  int next = 0;  // warp-uniform: next job to hand out
  int res = 0;
  bool active = false;
  V3 origin = v3(0.f, 0.f, 0.f), dir = v3(0.f, 0.f, 1.f), ad = v3(0.f, 0.f, 1.f);
  float dist = 0.f, diam = 0.f, stop = 0.f;
  bool check = false;
  float4 acc = f4(0.f, 0.f, 0.f, 0.f);
  // Software-pipelined like trace_cone_pipe: a lane computes its next step
  // (position, lod, empty-space test with its occupancy load) while the
  // current step's texture fetches are in flight, and issues the next
  // step's fetches as soon as the current one is added.  Same samples, same
  // arithmetic as trace_cone.
  float mip = 0.f;
  bool live = false;
  Taps t;
  for (;;) {
    const unsigned need = __ballot_sync(0xffffffffu, !active);
    if (need && next < n_jobs) {
      const int job = next + __popc(need & ((1u << lane) - 1u));
      if (!active && job < n_jobs) {
        const int jo = fw.order[job];
        const int k = jo / nq, q = jo - k * nq;
        res = q * K + k;
        const float4 jb = fw.job[jo];
        dir = v3(jb.x, jb.y, jb.z);
        stop = jb.w;
        origin = v3(fw.origin[q][0], fw.origin[q][1], fw.origin[q][2]);
        ad = vabs(dir);
        dist = dist1;
        diam = diam1;
        check = !march_sane(origin, dir, stop);
        acc = f4(0.f, 0.f, 0.f, 0.f);
        active = dist < stop;
        if (!active) {
          fw.far[res] = acc;
        } else {
          const V3 sp = march_pos(origin, dir, dist);
          mip = cone_lod(diam * cube_res);
          live = !(kSkipEmptyRGBA && m.skip_empty && mip < kSkipMaxLod && sample_empty(m, sp, mip)) &&
                 !(check && !u_sane(sp));
          if (live) issue_taps<false>(m, sp, octant(dir), ad, mip, t);
        }
      }
      next += __popc(need);
    }
    if (!__any_sync(0xffffffffu, active)) break;
    if (active) {
      const float step = fmaxf(diam * 0.5f, voxel_size);
      const float dist_n = dist + step;
      const float diam_n = dist_n * ap;
      const V3 sp_n = march_pos(origin, dir, dist_n);
      const bool more = dist_n < stop;
      const float mip_n = cone_lod(diam_n * cube_res);
      const bool live_n = more &&
                          !(kSkipEmptyRGBA && m.skip_empty && mip_n < kSkipMaxLod && sample_empty(m, sp_n, mip_n)) &&
                          !(check && !u_sane(sp_n));
      if (live) acc = fma4(combine_taps(t, ad, mip), 1.0f - acc.w, acc);
      if (!(acc.w < 1.0f) || !more) {
        fw.far[res] = acc;
        active = false;
      } else {
        dist = dist_n;
        diam = diam_n;
        mip = mip_n;
        live = live_n;
        if (live) issue_taps<false>(m, sp_n, octant(dir), ad, mip, t);
      }
    }
  }
}

// trace_diffuse with the group's far fields (far: this group's K results):
// each cone takes its first sample (step 0 of trace_cone) itself, then the
// far field behind it.
__device__ V3 trace_diffuse_shared(const MapSet& m, int cone_set, V3 origin, V3 n, const float4* far) {
  const V3 o1 = normalize(tangent(n));
  const V3 o2 = normalize(cross(o1, n));
  const int K = cone_set == VCT_CONES_SIX60 ? 6 : 9;
  const ConeStep e = m.sched->cone[cone_set].step[0];
  float4 acc = f4(0.f, 0.f, 0.f, 0.f);
  VCT_UNROLL_N(VCT_FIRST_UNROLL)
  for (int k = 0; k < K; ++k) {
    float ap;
    const V3 dir = normalize(diffuse_dir(cone_set, m.sched->ring, n, o1, o2, k, ap));
    // (the origin is a surface point inside the grid and the first step
    // three voxels: the sample position is sane, and one beyond the grid's
    // exit margin reads border texels, 0, as the unshortened march would)
    float4 c = cone_first<false>(m, origin, dir, e);
    if (c.w < 1.0f) c = fma4(far[k], 1.0f - c.w, c);
    acc = acc + c;
  }
  return v3(acc.x, acc.y, acc.z) * (1.0f / (float)K);
}

// Shades pixel (px, py) of one batch scene's frame (main,
// voxel_cone_tracing.frag:246-275): texture unit, anisotropic RGBA8 maps.
template <bool SHARE = false>
__device__ __forceinline__ void trace_px(const SceneParams& sp, const CameraParams& cp, const MapSet& m,
                                         const TraceParams& tp, const float4* __restrict__ gb_pos,
                                         const float4* __restrict__ gb_nrm, uchar4* __restrict__ frame, int px,
                                         int py, const float4* far = nullptr) {
  if (px >= cp.W || py >= cp.H) return;
  const size_t p = (size_t)py * cp.W + px;
  float4 out = f4(0.15f, 0.25f, 0.25f, 1.0f);  // glClearColor, renderer.cpp:398
  const float4 g0 = gb_pos[p], g1 = gb_nrm[p];
  if (__float_as_uint(g1.w) != 0xffffffffu) {
    const V3 world = v3(g0.x, g0.y, g0.z);
    const V3 nrm = v3(g1.x, g1.y, g1.z);
    const vct_material_data& mat = sp.materials[__float_as_uint(g0.w)];
    const V3 pos = v3(world.x / sp.cube_size, world.y / sp.cube_size, world.z / sp.cube_size) * 0.5f +
                   v3(0.5f, 0.5f, 0.5f);
    // within_cube(pos, 0) (:61-64, 250): a fragment outside returns without
    // writing; the pixel keeps the clear colour.
    if (fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f) {
      const V3 cam = v3(cp.cam_pos[0], cp.cam_pos[1], cp.cam_pos[2]);
      const V3 view_dir = normalize(world - cam);
      V3 fd = v3(0.f, 0.f, 0.f), fdir = v3(0.f, 0.f, 0.f), fs = v3(0.f, 0.f, 0.f);
      if (tp.enable_diffuse) {
        if (tp.diffuse_in) {
          const float4 d = tp.diffuse_in[p];
          fd = mulv(mat3v(mat.diffuse), v3(d.x, d.y, d.z));
        } else if (SHARE && far) {
          fd = mulv(mat3v(mat.diffuse), trace_diffuse_shared(m, tp.cone_set, pos, nrm, far));
        } else {
          fd = mulv(mat3v(mat.diffuse), trace_diffuse<false>(m, tp.cone_set, pos, nrm));
        }
      }
      if (tp.enable_direct)
        fdir = direct_light<false>(sp, m, tp.enable_shadow, mat, pos, nrm, view_dir, nullptr, 0);
      const float sap = specular_aperture(mat.shininess);
      if (tp.enable_specular) {
        const V3 sd = normalize(reflect(-view_dir, nrm));
        const float4 c = trace_cone<VCT_SAMPLER_HW, false, VCT_STORAGE_RGBA8>(m, pos, sd, sap, kMaxDistance);
        fs = mulv(mat3v(mat.specular), v3(c.x, c.y, c.z));
      }
      V3 f = fs + fd + fdir;
      if (refracts(mat) && tp.enable_specular) {
        const V3 rd = refract(view_dir, nrm, 1.0f / mat.ior);
        const float4 c = trace_cone<VCT_SAMPLER_HW, false, VCT_STORAGE_RGBA8>(m, pos, rd, sap, kMaxDistance);
        const V3 tr = mulv(mat3v(mat.transmittance), v3(c.x, c.y, c.z));
        f = tr * (1.0f - mat.dissolve) + f * mat.dissolve;
      }
      out = f4(f.x, f.y, f.z, 1.0f);
    }
  }
  frame[p] = make_uchar4(unorm8(out.x), unorm8(out.y), unorm8(out.z), unorm8(out.w));
}

// The voxel debug view (:253-257): one lookup a pixel.
template <int SAMPLER, bool ISO, int STORAGE>
__global__ void __launch_bounds__(256) k_view(SceneParams sp, CameraParams cp, const __grid_constant__ MapSet m,
                                              TraceParams tp, const float4* __restrict__ gb_pos,
                                              const float4* __restrict__ gb_nrm, uchar4* __restrict__ frame,
                                              float4* __restrict__ frame_f32) {
  const int px = blockIdx.x * 16 + (threadIdx.x & 15), py = blockIdx.y * 16 + (threadIdx.x >> 4);
  if (px >= cp.W || py >= cp.H) return;
  const size_t p = (size_t)py * cp.W + px;
  float4 out = f4(0.15f, 0.25f, 0.25f, 1.0f);  // glClearColor, renderer.cpp:398
  if (__float_as_uint(gb_nrm[p].w) != 0xffffffffu) {
    const float4 g0 = gb_pos[p];
    const V3 pos = v3(g0.x / sp.cube_size, g0.y / sp.cube_size, g0.z / sp.cube_size) * 0.5f + v3(0.5f, 0.5f, 0.5f);
    // within_cube(pos, 0) (:61-64, 250): a fragment outside returns without
    // writing; the pixel keeps the clear colour.
    if (fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f) {
      // (map 6: the isotropic chain of VCT_MIP_BOTH; no such map otherwise)
      out = f4(0.f, 0.f, 0.f, 0.f);
      if (tp.view_voxel_dir >= 0 && (tp.view_voxel_dir <= 5 || (tp.view_voxel_dir == 6 && m.nmaps == 7))) {
        const int d = ISO ? 0 : tp.view_voxel_dir;
        out = sample_voxel<SAMPLER, ISO, STORAGE>(m, pos, d, d, d, v3(1.f, 0.f, 0.f), fmaxf(tp.view_voxel_lod, 0.0f));
      }
    }
  }
  frame[p] = make_uchar4(unorm8(out.x), unorm8(out.y), unorm8(out.z), unorm8(out.w));
  if (frame_f32) frame_f32[p] = out;
}

// A frame with the FP32 software sampler (main, :246-275).  A step of a cone
// is 48 texel loads and their arithmetic, so a pixel's cones one after the
// other are a long serial chain and a small frame leaves most of the chip
// idle: a CTA takes an 8x4-pixel block with a warp per cone -- the diffuse
// cones, the specular (and refracted) one, the lights' shadow cones shared by
// up to kExactLights warps -- and its first warp puts them together.
// 320x180, 64^3, one light (GB300, the trace alone): 1741 us with a thread per pixel
// (255 registers, 8 warps an SM), 958 as here at 128 registers, 700 at 48,
// 647 at 40 (it spills 0.8 KB; more resident warps are worth it).  Bound by
// instructions (unpacking and weighting texels: ALU pipe 56%).
constexpr int kExactLights = 2;
template <bool ISO, int STORAGE>
__global__ void __launch_bounds__((9 + 1 + kExactLights) * 32, 4)
    k_trace_exact(SceneParams sp, CameraParams cp, const __grid_constant__ MapSet m, TraceParams tp, int diffuse_warps,
                  int light_warps, const float4* __restrict__ gb_pos, const float4* __restrict__ gb_nrm,
                  uchar4* __restrict__ frame, float4* __restrict__ frame_f32) {
  __shared__ float s_cone[11][3][32];  // 0-8: the diffuse cones, 9: specular, 10: refracted
  __shared__ float s_occ[kMaxLights][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int px = blockIdx.x * 8 + (lane & 7), py = blockIdx.y * 4 + (lane >> 3);
  const size_t p = (size_t)py * cp.W + px;
  const bool inside = px < cp.W && py < cp.H;
  bool valid = false;
  float4 g0 = f4(0.f, 0.f, 0.f, 0.f);
  V3 pos = v3(0.f, 0.f, 0.f), nrm = v3(0.f, 0.f, 1.f);
  if (inside) {
    const float4 g1 = gb_nrm[p];
    if (__float_as_uint(g1.w) != 0xffffffffu) {
      g0 = gb_pos[p];
      pos = v3(g0.x / sp.cube_size, g0.y / sp.cube_size, g0.z / sp.cube_size) * 0.5f + v3(0.5f, 0.5f, 0.5f);
      nrm = v3(g1.x, g1.y, g1.z);
      valid = fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f;  // within_cube, :250
    }
  }
  const int nl = min(max(sp.n_lights, 0), kMaxLights);
  const vct_material_data& mat = sp.materials[valid ? __float_as_uint(g0.w) : 0u];
  const V3 view_dir = normalize(v3(g0.x, g0.y, g0.z) - v3(cp.cam_pos[0], cp.cam_pos[1], cp.cam_pos[2]));
  auto keep = [&](int slot, float4 c) {
    s_cone[slot][0][lane] = c.x;
    s_cone[slot][1][lane] = c.y;
    s_cone[slot][2][lane] = c.z;
  };
  if (valid) {
    const int r = w - diffuse_warps;
    if (r > 0) {
      for (int i = r - 1; i < nl; i += light_warps) {
        V3 ld;
        float d;
        light_dir(sp, i, pos, ld, d);
        s_occ[i][lane] = m.skip_empty ? trace_shadow<VCT_SAMPLER_EXACT, ISO, STORAGE, false, true>(
                                            m, m.sched->shadow.group, pos, ld, d)
                                      : trace_shadow<VCT_SAMPLER_EXACT, ISO, STORAGE, false, false>(
                                            m, m.sched->shadow.group, pos, ld, d);
      }
    } else {
      // a diffuse cone, or the specular one and, of transparent materials, the refracted one
      int slot = w;
      V3 dir;
      float ap;
      if (r < 0) {
        const V3 o1 = normalize(tangent(nrm));
        const V3 o2 = normalize(cross(o1, nrm));
        dir = diffuse_dir(tp.cone_set, m.sched->ring, nrm, o1, o2, w, ap);
      } else {
        slot = 9;
        dir = normalize(reflect(-view_dir, nrm));
        ap = specular_aperture(mat.shininess);
      }
      const int passes = r < 0 ? 1 : (!tp.enable_specular ? 0 : (refracts(mat) ? 2 : 1));
#pragma unroll 1
      for (int pass = 0; pass < passes; ++pass) {
        if (pass) dir = refract(view_dir, nrm, 1.0f / mat.ior);
        keep(slot + pass, trace_cone<VCT_SAMPLER_EXACT, ISO, STORAGE>(m, pos, dir, ap, kMaxDistance));
      }
    }
  }
  __syncthreads();
  if (w != 0 || !inside) return;
  float4 out = f4(0.15f, 0.25f, 0.25f, 1.0f);  // glClearColor, renderer.cpp:398
  if (valid) {
    auto cone = [&](int slot) { return v3(s_cone[slot][0][lane], s_cone[slot][1][lane], s_cone[slot][2][lane]); };
    V3 fd = v3(0.f, 0.f, 0.f), fdir = v3(0.f, 0.f, 0.f), fs = v3(0.f, 0.f, 0.f);
    if (tp.enable_diffuse) {
      V3 d;
      if (tp.diffuse_in) {
        const float4 q = tp.diffuse_in[p];
        d = v3(q.x, q.y, q.z);
      } else {
        d = cone(0);
        for (int k = 1; k < diffuse_warps; ++k) d = d + cone(k);
        d = d * (1.0f / (float)diffuse_warps);
      }
      fd = mulv(mat3v(mat.diffuse), d);
    }
    if (tp.enable_direct)
      fdir = direct_light<true>(sp, m, tp.enable_shadow, mat, pos, nrm, view_dir, &s_occ[0][lane], 32);
    if (tp.enable_specular) fs = mulv(mat3v(mat.specular), cone(9));
    V3 f = fs + fd + fdir;
    if (refracts(mat) && tp.enable_specular) {
      const V3 tr = mulv(mat3v(mat.transmittance), cone(10));
      f = tr * (1.0f - mat.dissolve) + f * mat.dissolve;
    }
    out = f4(f.x, f.y, f.z, 1.0f);
  }
  frame[p] = make_uchar4(unorm8(out.x), unorm8(out.y), unorm8(out.z), unorm8(out.w));
  if (frame_f32) frame_f32[p] = out;
}

// One pixel of the one-launch batch tracers: the warp (a block of kShareW x 2 groups, its
// rows starting at an even frame row; share_tile_px) first picks each group's
// representative (its first pixel, row by row, whose diffuse cones are
// traced) and the pixels that share with it, marches the groups' far fields
// together (far_fields), then shades its pixels (trace_px).  Called by
// all 32 lanes of a warp together; fw is the warp's shared-memory block.
__device__ __forceinline__ void trace_px_share(const SceneParams& sp, const CameraParams& cp, const MapSet& m,
                                               const TraceParams& tp, const float4* __restrict__ gb_pos,
                                               const float4* __restrict__ gb_nrm, uchar4* __restrict__ frame,
                                               int px, int py, FarWarp& fw) {
  const int lane = threadIdx.x & 31;
  bool valid = false;
  V3 pos = v3(0.f, 0.f, 0.f), nrm = v3(0.f, 0.f, 1.f);
  if (px < cp.W && py < cp.H) {
    const size_t p = (size_t)py * cp.W + px;
    const float4 g0 = gb_pos[p], g1 = gb_nrm[p];
    if (__float_as_uint(g1.w) != 0xffffffffu) {
      pos = v3(g0.x / sp.cube_size, g0.y / sp.cube_size, g0.z / sp.cube_size) * 0.5f + v3(0.5f, 0.5f, 0.5f);
      nrm = v3(g1.x, g1.y, g1.z);
      // the pixels whose diffuse cones trace_px traces (within_cube, :250)
      valid = fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f;
    }
  }
  valid = valid && tp.enable_diffuse && tp.view_voxel_dir >= 7 && !tp.diffuse_in;
  int rep;
  const bool share = group_share(m.N, valid, pos, nrm, rep);
  const int K = tp.cone_set == VCT_CONES_SIX60 ? 6 : 9;
  const unsigned repmask = __ballot_sync(0xffffffffu, valid && rep == lane);
  const int slot = __popc(repmask & ((1u << rep) - 1u));
  if (valid && rep == lane) {
    fw.origin[slot][0] = pos.x;
    fw.origin[slot][1] = pos.y;
    fw.origin[slot][2] = pos.z;
    fw.normal[slot][0] = nrm.x;
    fw.normal[slot][1] = nrm.y;
    fw.normal[slot][2] = nrm.z;
  }
  __syncwarp();
  // the second step of the march schedule (trace_cone's recurrence)
  const float ap = tp.cone_set == VCT_CONES_SIX60 ? kSixAperture : kTan22_5;
  const float voxel_size = 1.0f / (float)m.N;
  const float dist0 = 3.0f * voxel_size;
  const float dist1 = dist0 + fmaxf(dist0 * ap * 0.5f, voxel_size);
  if (repmask) far_fields(m, fw, tp.cone_set, __popc(repmask), dist1, dist1 * ap);
  __syncwarp();
  trace_px<true>(sp, cp, m, tp, gb_pos, gb_nrm, frame, px, py, share ? fw.far + slot * K : nullptr);
  __syncwarp();  // fw is free for the warp's next use
}

// One pixel of a batch scene.  Called, not inlined, from the tile loop of
// k_trace_batch: inlined into a loop, the shading's loop-invariant loads
// (scene constants, texture handles) are hoisted out of the loop and held in
// registers across all tiles, which spills the march loop (measured: 4 KB of
// spill code against 0.2 KB for the one-scene kernel).
#ifdef VCT_TRACE_BATCH_INLINE
#define VCT_BATCH_PX_FN __forceinline__
#else
#define VCT_BATCH_PX_FN __noinline__
#endif
// The current scene of a k_trace_batch CTA, read by trace_batch_px at fixed
// shared-memory addresses.
__shared__ BatchScene s_batch_scene;
__shared__ CameraParams s_batch_cam;

__device__ VCT_BATCH_PX_FN void trace_batch_px(const float4* __restrict__ gb_pos, const float4* __restrict__ gb_nrm,
                                            uchar4* __restrict__ frame, int px, int py) {
  trace_px(s_batch_scene.sp, s_batch_cam, s_batch_scene.ms, s_batch_scene.tp, gb_pos, gb_nrm, frame, px, py);
}

// trace_px_share on the CTA's current batch scene (k_trace_batch_share);
// called, not inlined, for the same reason as trace_batch_px.
__device__ VCT_BATCH_PX_FN void trace_batch_px_share(const float4* __restrict__ gb_pos,
                                                  const float4* __restrict__ gb_nrm, uchar4* __restrict__ frame,
                                                  int px, int py, FarWarp& fw) {
  trace_px_share(s_batch_scene.sp, s_batch_cam, s_batch_scene.ms, s_batch_scene.tp, gb_pos, gb_nrm, frame, px, py,
                 fw);
}

// The 16x16 tiles of every scene of a batch in one persistent launch.  With
// w.queue a CTA takes its next tile from an atomic counter (uneven scenes
// balance across SMs); without, tiles are strided by the grid.  The CTA
// keeps its current scene's descriptor and camera in shared memory, so the
// shading code addresses them at fixed offsets (as kernel parameters are in
// the one-scene kernel) instead of holding pointers in registers.
__global__ void __launch_bounds__(256, kTraceBatchMinBlocks) k_trace_batch(BatchWork w, BatchBuffers bb) {
  __shared__ uint32_t s_next;
  __shared__ int s_cur;
  BatchScene& s_sc = s_batch_scene;
  CameraParams& s_cam = s_batch_cam;
  static_assert(sizeof(BatchScene) % 4 == 0 && sizeof(CameraParams) % 4 == 0, "word copies");
  uint32_t g = blockIdx.x;
  if (threadIdx.x == 0) s_cur = -1;
  if (w.queue) {
    if (threadIdx.x == 0) s_next = atomicAdd(w.queue, 1u);
    __syncthreads();
    g = s_next;
  }
  __syncthreads();
  while (g < w.total) {
    const int s = batch_scene_of(w, g);
    if (s != s_cur) {  // CTA-uniform
      __syncthreads();  // the previous tile is done with the old scene
      const uint32_t* src = reinterpret_cast<const uint32_t*>(w.scenes + s);
      for (int i = threadIdx.x; i < (int)(sizeof(BatchScene) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&s_sc)[i] = __ldg(src + i);
      const uint32_t* csrc = reinterpret_cast<const uint32_t*>(w.cams + s);
      for (int i = threadIdx.x; i < (int)(sizeof(CameraParams) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&s_cam)[i] = __ldg(csrc + i);
      __syncthreads();
      if (threadIdx.x == 0) s_cur = s;
    }
    const uint32_t lt = g - __ldg(w.prefix + s), tiles_x = (uint32_t)(s_sc.W + 15) / 16;
    trace_batch_px(bb.rb.gb_pos + s_sc.px_base, bb.rb.gb_nrm + s_sc.px_base, bb.frame + s_sc.px_base,
                   (int)(lt % tiles_x) * 16 + (threadIdx.x & 15), (int)(lt / tiles_x) * 16 + (threadIdx.x >> 4));
    if (w.queue) {
      __syncthreads();  // every thread has read s_next
      if (threadIdx.x == 0) s_next = atomicAdd(w.queue, 1u);
      __syncthreads();
      g = s_next;
    } else {
      g += gridDim.x;
    }
  }
}

// k_trace_batch with shared far fields (the batch's far_share): every 16x16
// tile is eight 8x4 warps, as in k_march and k_shade, so each scene's frame equals
// a Renderer's with far_share 1.  Anisotropic maps (the batch's).
#ifndef VCT_TRACE_BATCH_SHARE_MIN_BLOCKS
#define VCT_TRACE_BATCH_SHARE_MIN_BLOCKS 4
#endif
constexpr int kTraceBatchShareMinBlocks = VCT_TRACE_BATCH_SHARE_MIN_BLOCKS;
__global__ void __launch_bounds__(256, kTraceBatchShareMinBlocks) k_trace_batch_share(BatchWork w, BatchBuffers bb) {
  __shared__ FarWarp s_far[8];
  __shared__ uint32_t s_next;
  __shared__ int s_cur;
  BatchScene& s_sc = s_batch_scene;
  CameraParams& s_cam = s_batch_cam;
  static_assert(sizeof(BatchScene) % 4 == 0 && sizeof(CameraParams) % 4 == 0, "word copies");
  uint32_t g = blockIdx.x;
  if (threadIdx.x == 0) s_cur = -1;
  if (w.queue) {
    if (threadIdx.x == 0) s_next = atomicAdd(w.queue, 1u);
    __syncthreads();
    g = s_next;
  }
  __syncthreads();
  while (g < w.total) {
    const int s = batch_scene_of(w, g);
    if (s != s_cur) {  // CTA-uniform
      __syncthreads();  // the previous tile is done with the old scene
      const uint32_t* src = reinterpret_cast<const uint32_t*>(w.scenes + s);
      for (int i = threadIdx.x; i < (int)(sizeof(BatchScene) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&s_sc)[i] = __ldg(src + i);
      const uint32_t* csrc = reinterpret_cast<const uint32_t*>(w.cams + s);
      for (int i = threadIdx.x; i < (int)(sizeof(CameraParams) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&s_cam)[i] = __ldg(csrc + i);
      __syncthreads();
      if (threadIdx.x == 0) s_cur = s;
    }
    const uint32_t lt = g - __ldg(w.prefix + s), tiles_x = (uint32_t)(s_sc.W + 15) / 16;
    int px, py;
    share_tile_px((int)(lt % tiles_x) * 16, (int)(lt / tiles_x) * 16, px, py);
    trace_batch_px_share(bb.rb.gb_pos + s_sc.px_base, bb.rb.gb_nrm + s_sc.px_base, bb.frame + s_sc.px_base, px, py,
                         s_far[threadIdx.x >> 5]);
    if (w.queue) {
      __syncthreads();  // every thread has read s_next
      if (threadIdx.x == 0) s_next = atomicAdd(w.queue, 1u);
      __syncthreads();
      g = s_next;
    } else {
      g += gridDim.x;
    }
  }
}

// One CTA per 16x16 tile of every scene of the batch, in one launch
// (BatchShape::trace_ctas_per_sm 0).  Without a tile loop the shading is
// inlined, as in the one-scene kernels, while the scene's descriptor and
// camera come from shared memory: a CTA looks up its scene, copies them
// there and traces its tile.
template <bool SHARE>
__global__ void __launch_bounds__(256, SHARE ? kTraceBatchShareMinBlocks : kTraceBatchMinBlocks)
    k_trace_batch_tiles(BatchWork w, BatchBuffers bb) {
  __shared__ FarWarp s_far[SHARE ? 8 : 1];
  BatchScene& s_sc = s_batch_scene;
  CameraParams& s_cam = s_batch_cam;
  const uint32_t g = blockIdx.x;
  const int s = batch_scene_of_warp(w, g);  // every warp finds it: no barrier before the copy
  const uint32_t* src = reinterpret_cast<const uint32_t*>(w.scenes + s);
  for (int i = threadIdx.x; i < (int)(sizeof(BatchScene) / 4); i += blockDim.x)
    reinterpret_cast<uint32_t*>(&s_sc)[i] = __ldg(src + i);
  const uint32_t* csrc = reinterpret_cast<const uint32_t*>(w.cams + s);
  for (int i = threadIdx.x; i < (int)(sizeof(CameraParams) / 4); i += blockDim.x)
    reinterpret_cast<uint32_t*>(&s_cam)[i] = __ldg(csrc + i);
  __syncthreads();
  const uint32_t lt = g - __ldg(w.prefix + s), tiles_x = (uint32_t)(s_sc.W + 15) / 16;
  int px, py;
  share_tile_px((int)(lt % tiles_x) * 16, (int)(lt / tiles_x) * 16, px, py);
  const float4* gp = bb.rb.gb_pos + s_sc.px_base;
  const float4* gn = bb.rb.gb_nrm + s_sc.px_base;
  uchar4* fr = bb.frame + s_sc.px_base;
  if constexpr (SHARE)
    trace_px_share(s_sc.sp, s_cam, s_sc.ms, s_sc.tp, gp, gn, fr, px, py, s_far[threadIdx.x >> 5]);
  else
    trace_px(s_sc.sp, s_cam, s_sc.ms, s_sc.tp, gp, gn, fr, px, py);
}

template <int SAMPLER, bool ISO, int STORAGE>
cudaError_t run_view(const SceneParams& sp, const CameraParams& cp, const MapSet& ms, const TraceParams& tp,
                     const float4* gb_pos, const float4* gb_nrm, uchar4* frame, float4* frame_f32, cudaStream_t st) {
  const dim3 grid((cp.W + 15) / 16, (cp.H + 15) / 16);
  k_view<SAMPLER, ISO, STORAGE><<<grid, 256, 0, st>>>(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32);
  return cudaGetLastError();
}

template <bool ISO, int STORAGE>
cudaError_t run_exact(const SceneParams& sp, const CameraParams& cp, const MapSet& ms, const TraceParams& tp,
                      const float4* gb_pos, const float4* gb_nrm, uchar4* frame, float4* frame_f32, cudaStream_t st) {
  if (tp.view_voxel_dir < 7)
    return run_view<VCT_SAMPLER_EXACT, ISO, STORAGE>(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, st);
  const int nl = std::min(std::max(sp.n_lights, 0), kMaxLights);
  const int diffuse = tp.enable_diffuse && !tp.diffuse_in ? (tp.cone_set == VCT_CONES_SIX60 ? 6 : 9) : 0;
  const int lights = tp.enable_direct && tp.enable_shadow ? std::min(nl, kExactLights) : 0;
  const dim3 grid((cp.W + 7) / 8, (cp.H + 3) / 4);
  k_trace_exact<ISO, STORAGE><<<grid, (diffuse + 1 + lights) * 32, 0, st>>>(sp, cp, ms, tp, diffuse, lights, gb_pos,
                                                                            gb_nrm, frame, frame_f32);
  return cudaGetLastError();
}

// Training targets of the learned term: trace_diffuse (texture-unit sampler)
// at each sample's texture-space position and normal (rows of 12 floats;
// writes columns 9..11).
template <bool ISO>
__global__ void __launch_bounds__(256) k_trace_points(MapSet m, int cone_set, float* __restrict__ samples, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float* q = samples + (size_t)i * 12;
  const V3 pos = v3(q[0], q[1], q[2]), nrm = v3(q[3], q[4], q[5]);
  const V3 d = trace_diffuse<ISO>(m, cone_set, pos, nrm);
  q[9] = d.x;
  q[10] = d.y;
  q[11] = d.z;
}

// The judge of the learned diffuse term (launch_judge_diffuse): one pixel
// per stride x stride tile, the same visibility and within_cube test as
// trace_px, the cones of trace_diffuse with the texture unit against the
// network's prediction of them.  A CTA judges 32 pixels with one thread per
// (pixel, cone), so that the few judged pixels still fill the GPU; the
// cones of a pixel are summed in trace_diffuse's order.
constexpr int kJudgePixels = 32;
template <bool ISO>
__global__ void __launch_bounds__(kJudgePixels * 9) k_judge_diffuse(SceneParams sp, MapSet m, TraceParams tp, int W,
                                                                    int H, const float4* __restrict__ gb_pos,
                                                                    const float4* __restrict__ gb_nrm,
                                                                    const float4* __restrict__ net, int stride, int ox,
                                                                    int oy, int tw, int n_judged,
                                                                    FrameStatus* __restrict__ status) {
  __shared__ float4 s_cone[9][kJudgePixels];
  const int j = threadIdx.x % kJudgePixels, k = threadIdx.x / kJudgePixels;
  const int K = tp.cone_set == VCT_CONES_SIX60 ? 6 : 9;
  const int i = blockIdx.x * kJudgePixels + j;
  bool judged = false;
  size_t p = 0;
  if (i < n_judged) {
    const int px = (i % tw) * stride + ox, py = (i / tw) * stride + oy;
    if (px < W && py < H) {
      p = (size_t)py * W + px;
      const float4 g0 = gb_pos[p], g1 = gb_nrm[p];
      if (__float_as_uint(g1.w) != 0xffffffffu) {
        const V3 pos =
            v3(g0.x / sp.cube_size, g0.y / sp.cube_size, g0.z / sp.cube_size) * 0.5f + v3(0.5f, 0.5f, 0.5f);
        judged = fabsf(pos.x) < 1.0f && fabsf(pos.y) < 1.0f && fabsf(pos.z) < 1.0f;
        if (judged && k < K) {
          const V3 n = v3(g1.x, g1.y, g1.z);
          const V3 o1 = normalize(tangent(n));
          const V3 o2 = normalize(cross(o1, n));
          float ap;
          const V3 d = diffuse_dir(tp.cone_set, m.sched->ring, n, o1, o2, k, ap);
          s_cone[k][j] = trace_cone<VCT_SAMPLER_HW, ISO, VCT_STORAGE_RGBA8>(m, pos, d, ap, kMaxDistance);
        }
      }
    }
  }
  __syncthreads();
  if (k != 0) return;  // one warp sums
  float e = 0.0f;
  uint32_t n = 0;
  if (judged) {
    float4 acc = f4(0.f, 0.f, 0.f, 0.f);
    for (int c = 0; c < K; ++c) acc = acc + s_cone[c][j];
    const V3 d = v3(acc.x, acc.y, acc.z) * (1.0f / (float)K);
    const float4 q = net[p];
    e = (d.x - q.x) * (d.x - q.x) + (d.y - q.y) * (d.y - q.y) + (d.z - q.z) * (d.z - q.z);
    n = 1;
  }
  for (int o = 16; o > 0; o >>= 1) {
    e += __shfl_xor_sync(0xffffffffu, e, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  if (threadIdx.x == 0 && n) {
    atomicAdd(&status->judge_sse, e);
    atomicAdd(&status->judge_n, n);
  }
}

}  // namespace

cudaError_t launch_judge_diffuse(const SceneParams& sp, const CameraParams& cp, const MapSet& ms, const TraceParams& tp,
                                 const float4* gb_pos, const float4* gb_nrm, const float4* net, int stride, int ox,
                                 int oy, FrameStatus* status, cudaStream_t st) {
  if (stride < 1) return cudaSuccess;
  const int tw = (cp.W - ox + stride - 1) / stride, th = (cp.H - oy + stride - 1) / stride;
  if (tw <= 0 || th <= 0) return cudaSuccess;
  const int n_judged = tw * th;
  const unsigned blocks = (unsigned)((n_judged + kJudgePixels - 1) / kJudgePixels);
  if (tp.mip_mode == VCT_MIP_ISO)
    k_judge_diffuse<true><<<blocks, kJudgePixels * 9, 0, st>>>(sp, ms, tp, cp.W, cp.H, gb_pos, gb_nrm, net, stride, ox,
                                                              oy, tw, n_judged, status);
  else
    k_judge_diffuse<false><<<blocks, kJudgePixels * 9, 0, st>>>(sp, ms, tp, cp.W, cp.H, gb_pos, gb_nrm, net, stride,
                                                               ox, oy, tw, n_judged, status);
  return cudaGetLastError();
}

cudaError_t launch_trace_points(const SceneParams&, const MapSet& ms, int mip_mode, int cone_set, float* samples,
                                int n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (mip_mode == VCT_MIP_ISO) k_trace_points<true><<<grid, 256, 0, st>>>(ms, cone_set, samples, n);
  else k_trace_points<false><<<grid, 256, 0, st>>>(ms, cone_set, samples, n);
  return cudaGetLastError();
}

cudaError_t launch_trace_batch(const BatchWork& tiles, const BatchBuffers& bb, const BatchShape& shape, int sms,
                               cudaStream_t st, int* launches, bool share) {
  if (!tiles.total) return cudaSuccess;
  BatchWork w = tiles;
  if (shape.trace_ctas_per_sm == 0) {  // one CTA per tile
    if (share) k_trace_batch_tiles<true><<<tiles.total, 256, 0, st>>>(w, bb);
    else k_trace_batch_tiles<false><<<tiles.total, 256, 0, st>>>(w, bb);
    if (launches) ++*launches;
    return cudaGetLastError();
  }
  if (!shape.trace_dynamic) w.queue = nullptr;
  else {
    cudaError_t e = cudaMemsetAsync(w.queue, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
  }
  if (share) {
    const int per_sm = std::min(std::max(shape.trace_ctas_per_sm, 1), kTraceBatchShareMinBlocks);
    const unsigned grid = (unsigned)std::max(1, std::min<int>(sms * per_sm, (int)tiles.total));
    k_trace_batch_share<<<grid, 256, 0, st>>>(w, bb);
    if (launches) ++*launches;
    return cudaGetLastError();
  }
  const int per_sm = std::min(std::max(shape.trace_ctas_per_sm, 1), kTraceBatchMinBlocks);
  const unsigned grid = (unsigned)std::max(1, std::min<int>(sms * per_sm, (int)tiles.total));
  k_trace_batch<<<grid, 256, 0, st>>>(w, bb);
  if (launches) ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_trace_px(const SceneParams& sp, const CameraParams& cp, const MapSet& ms, const TraceParams& tp,
                            const float4* gb_pos, const float4* gb_nrm, uchar4* frame, float4* frame_f32,
                            cudaStream_t st, int* launches) {
  if (launches) ++*launches;
  const bool iso = tp.mip_mode == VCT_MIP_ISO, rgba8 = ms.storage == VCT_STORAGE_RGBA8;
  if (tp.sampler == VCT_SAMPLER_EXACT) {
    auto run = iso ? (rgba8 ? run_exact<true, VCT_STORAGE_RGBA8> : run_exact<true, VCT_STORAGE_RGBA16F>)
                   : (rgba8 ? run_exact<false, VCT_STORAGE_RGBA8> : run_exact<false, VCT_STORAGE_RGBA16F>);
    return run(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, st);
  }
  auto run = iso ? run_view<VCT_SAMPLER_HW, true, VCT_STORAGE_RGBA8> : run_view<VCT_SAMPLER_HW, false, VCT_STORAGE_RGBA8>;
  return run(sp, cp, ms, tp, gb_pos, gb_nrm, frame, frame_f32, st);
}

}  // namespace vct
