// k_voxelize.cu -- the Voxelizer: replaces voxelize.vert/.geom/.frag and the
// level-0 clear of Renderer::voxelize (renderer.cpp:316-353).
//
// Pipeline (all stream-ordered, no host synchronisation):
//   1. k_bin<false>: every queued triangle -> the 8^3-voxel bricks its
//      (margin-expanded) box test says it may touch; per-brick counts.
//   2. exclusive scan of the counts -> per-brick list offsets.
//   3. k_bin<true>: scatter triangle ids into the per-brick lists.
//   4. k_bricks: resident CTAs take the bricks that have pairs (and the empty
//      ones that must be cleared) from a list the scan makes.  A CTA sets up
//      128 pairs in shared memory, decides coverage with the exact rule of the
//      selected mode, shades what is covered in FP32 (voxelize.frag:124-153),
//      adds fixed-point colour sums and counts into shared-memory
//      accumulators, and writes its whole brick of level 0 as RGBA8 or RGBA16F
//      through a surface -- level 0 is written exactly once.
//
// Coverage rules (the CPU oracle implements the same ones):
//   REF_RASTER2X -- the reference's method: dominant-axis projection
//     (voxelize.geom:27-51) rasterised on the 2N x 2N viewport
//     (renderer.cpp:339-340): vertices snapped to 1/256 sample pixel,
//     integer edge functions, top-left fill rule; sample depth = FP32
//     barycentric interpolation, voxel = int(N*(0.5*c+0.5)) (voxelize.frag
//     :156-157, truncation).
//   CONSERVATIVE -- exact separating-axis triangle/box test on vertices
//     snapped to 1/256 voxel (vct_cover.h), colour at the triangle point
//     closest to the voxel centre.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>
#include <climits>
#include <type_traits>

#include "vct_cover.h"
#include "vct_internal.h"
#include "vct_math.cuh"
#include "vct_mip.cuh"
#include "vct_snap.h"

namespace vct {
namespace {

#ifndef VCT_BRICK_THREADS
#define VCT_BRICK_THREADS 128
#endif
constexpr int kThreads = VCT_BRICK_THREADS;  // threads of a brick CTA
constexpr int kWarps = kThreads / 32;
#ifndef VCT_BRICK_ROUND
#define VCT_BRICK_ROUND 0
#endif
// Pairs per round of a brick CTA (0: one per thread); their triangle setups
// are the larger part of its shared memory.
constexpr int kRound = VCT_BRICK_ROUND > 0 ? VCT_BRICK_ROUND : kThreads;
static_assert(kRound % 32 == 0 && kRound <= kThreads, "round of whole warps, at most one pair per thread");
// Resident brick CTAs per SM the kernels are compiled for: 7 (72 registers,
// 26 to 28 KB of shared memory each with RGBA8), 5 where the attribute sums
// take 40 KB.  96-pair rounds at 8 per SM (64 registers) and 96-thread CTAs at
// 9 took the same or longer (512^3: 985 us of voxelization against 1006 and
// 1112), 64-pair rounds longer still.
template <int STORAGE>
constexpr int brick_min_blocks() {
  return STORAGE == kStorageAttr ? 5 : 7;
}
constexpr int kBrickVox = kBrick * kBrick * kBrick;
constexpr float kBinMargin = 0.25f;   // voxels; >> snapping and FP32 error
constexpr float kFix = 65535.0f;      // fixed-point scale of one contribution

// ------------------------------------------------------------ triangle load --
__device__ __forceinline__ int find_instance(const SceneParams& sp, uint32_t t) {
  int lo = 0, hi = (int)sp.n_instances - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (sp.inst[mid].tri_base <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

struct TriLoad {
  float g[3][3];   // grid-space positions (voxelize.vert:26), FP32 fixed order
  V3 n[3];         // normalize(NM * normal) (voxelize.vert:28)
  uint32_t mat;
  bool ok;
};

template <bool NORMALS>
__device__ __forceinline__ void load_tri(const SceneParams& sp, uint32_t t, TriLoad& tl) {
  const DevInstance& in = sp.inst[find_instance(sp, t)];
  const uint32_t lt = t - in.tri_base;
  tl.ok = true;
  for (int k = 0; k < 3; ++k) {
    // Indices and material ids of host-side meshes are checked when they are
    // loaded; those of caller-owned device meshes are clamped here (and
    // counted by the caller's entry point), so that no id reads out of bounds.
    const uint32_t vi = min(__ldg(in.indices + 3 * (size_t)lt + k), in.n_verts - 1u);
    const float4* vp = reinterpret_cast<const float4*>(in.verts + vi);
    const float4 a = __ldg(vp), b = __ldg(vp + 1);
    for (int r = 0; r < 3; ++r) {
      float w = xform_row(in.M, r, a.x, a.y, a.z);
      float gv = rdiv(w, sp.cube_size);
      tl.g[k][r] = gv;
      if (!(fabsf(gv) <= 64.0f)) tl.ok = false;
    }
    if (NORMALS) tl.n[k] = normalize(nm_mul(in.NM, a.w, b.x, b.y));
  }
  if (NORMALS) tl.mat = __ldg(sp.obj_material + min(__ldg(in.tri_obj + lt), sp.n_obj - 1u));
}

__device__ __forceinline__ void store_rec(TriRec& r, const TriLoad& tl) {
  r.q[0] = make_float4(tl.g[0][0], tl.g[0][1], tl.g[0][2], tl.g[1][0]);
  r.q[1] = make_float4(tl.g[1][1], tl.g[1][2], tl.g[2][0], tl.g[2][1]);
  r.q[2] = make_float4(tl.g[2][2], tl.n[0].x, tl.n[0].y, tl.n[0].z);
  r.q[3] = make_float4(tl.n[1].x, tl.n[1].y, tl.n[1].z, tl.n[2].x);
  r.q[4] = make_float4(tl.n[2].y, tl.n[2].z, __uint_as_float(tl.mat), 0.0f);
}
__device__ __forceinline__ void load_rec(const TriRec& r, TriLoad& tl) {
  const float4 a = r.q[0], b = r.q[1], c = r.q[2], d = r.q[3], e = r.q[4];
  tl.g[0][0] = a.x; tl.g[0][1] = a.y; tl.g[0][2] = a.z;
  tl.g[1][0] = a.w; tl.g[1][1] = b.x; tl.g[1][2] = b.y;
  tl.g[2][0] = b.z; tl.g[2][1] = b.w; tl.g[2][2] = c.x;
  tl.n[0] = v3(c.y, c.z, c.w);
  tl.n[1] = v3(d.x, d.y, d.z);
  tl.n[2] = v3(d.w, e.x, e.y);
  tl.mat = __float_as_uint(e.z);
  tl.ok = true;
}
// A listed triangle: from its record, or without records from the meshes.
template <bool REC>
__device__ __forceinline__ void fetch_tri(const SceneParams& sp, const TriRec* __restrict__ recs, uint32_t t,
                                          TriLoad& tl) {
  if constexpr (REC) load_rec(recs[t], tl);
  else load_tri<true>(sp, t, tl);
}

// ------------------------------------------------ conservative brick test --
// Triangle / axis-aligned box overlap in FP32 (box normals, plane, 9 edge
// axes).  Only used for binning, with boxes grown by kBinMargin, so FP32
// rounding can only add candidates.
__device__ bool tri_box_f32(const float v[3][3], const float c[3], const float h[3]) {
  float u[3][3];
  for (int k = 0; k < 3; ++k)
    for (int d = 0; d < 3; ++d) u[k][d] = v[k][d] - c[d];
  for (int d = 0; d < 3; ++d) {
    float mn = fminf(u[0][d], fminf(u[1][d], u[2][d])), mx = fmaxf(u[0][d], fmaxf(u[1][d], u[2][d]));
    if (mn > h[d] || mx < -h[d]) return false;
  }
  float f[3][3];
  for (int d = 0; d < 3; ++d) {
    f[0][d] = u[1][d] - u[0][d];
    f[1][d] = u[2][d] - u[1][d];
    f[2][d] = u[0][d] - u[2][d];
  }
  float n0 = f[0][1] * f[1][2] - f[0][2] * f[1][1];
  float n1 = f[0][2] * f[1][0] - f[0][0] * f[1][2];
  float n2 = f[0][0] * f[1][1] - f[0][1] * f[1][0];
  float dd = n0 * u[0][0] + n1 * u[0][1] + n2 * u[0][2];
  float rr = h[0] * fabsf(n0) + h[1] * fabsf(n1) + h[2] * fabsf(n2);
  if (fabsf(dd) > rr * 1.0001f + 1e-6f) return false;
  for (int e = 0; e < 3; ++e) {
    const float fx = f[e][0], fy = f[e][1], fz = f[e][2];
    float p0, p1, p2, r;
    p0 = -fz * u[0][1] + fy * u[0][2]; p1 = -fz * u[1][1] + fy * u[1][2]; p2 = -fz * u[2][1] + fy * u[2][2];
    r = h[1] * fabsf(fz) + h[2] * fabsf(fy);
    if (fminf(p0, fminf(p1, p2)) > r * 1.0001f || fmaxf(p0, fmaxf(p1, p2)) < -r * 1.0001f) return false;
    p0 = fz * u[0][0] - fx * u[0][2]; p1 = fz * u[1][0] - fx * u[1][2]; p2 = fz * u[2][0] - fx * u[2][2];
    r = h[0] * fabsf(fz) + h[2] * fabsf(fx);
    if (fminf(p0, fminf(p1, p2)) > r * 1.0001f || fmaxf(p0, fmaxf(p1, p2)) < -r * 1.0001f) return false;
    p0 = -fy * u[0][0] + fx * u[0][1]; p1 = -fy * u[1][0] + fx * u[1][1]; p2 = -fy * u[2][0] + fx * u[2][1];
    r = h[0] * fabsf(fy) + h[1] * fabsf(fx);
    if (fminf(p0, fminf(p1, p2)) > r * 1.0001f || fmaxf(p0, fmaxf(p1, p2)) < -r * 1.0001f) return false;
  }
  return true;
}

// May triangle v (voxel units) touch brick (bx, by, bz)?
__device__ __forceinline__ bool touches_brick(const float v[3][3], int bx, int by, int bz) {
  const int b3[3] = {bx, by, bz};
  float c[3], h[3];
  for (int d = 0; d < 3; ++d) {
    float lo = (float)(b3[d] * kBrick) - kBinMargin - (b3[d] == 0 ? 1.0f : 0.0f);
    float hi = (float)(b3[d] * kBrick + kBrick) + kBinMargin;
    c[d] = 0.5f * (lo + hi);
    h[d] = 0.5f * (hi - lo);
  }
  return tri_box_f32(v, c, h);
}

// One (triangle, candidate brick) pair of the binning passes.
template <bool FILL>
__device__ __forceinline__ void bin_one(const float v[3][3], int bx, int by, int bz, int nb, uint32_t t,
                                        uint32_t* count, uint32_t* cursor, uint32_t* __restrict__ list,
                                        uint32_t cap) {
  if (!touches_brick(v, bx, by, bz)) return;
  const uint32_t brick = ((uint32_t)bz * nb + by) * nb + bx;
  if (FILL) {
    uint32_t slot = atomicAdd(cursor + brick, 1u);
    if (slot < cap) list[slot] = t;
  } else {
    atomicAdd(count + brick, 1u);
  }
}

constexpr int kSoloBricks = 8;  // candidate bricks a lane bins on its own
constexpr int kBigSplit = 8;     // CTAs that share one large triangle
// Bin record of a triangle (counting pass -> filling pass): x = first
// candidate brick (10 bits per axis), y = bits 0-7 which of its (at most
// kSoloBricks) candidates passed the triangle/box test, bits 8-16 the
// candidate extents - 1 (3 bits per axis), bit 31 = bin it again in the
// filling pass (triangles the warp bins together).  Triangles of large-
// triangle records and rejected ones have no bricks here.
constexpr uint32_t kRecAgain = 1u << 31;

// Bins every triangle to the bricks it may touch.  A lane handles its own
// triangle when it has few candidate bricks.  A triangle with more
// candidates (room walls span 1024 bricks at 256^3) is recorded by the
// counting pass in `big` and binned by k_bin_big, which spreads each record
// over several CTAs; when the record list is full the warp bins it, the lanes
// splitting the candidate range.
// All 32 lanes of a warp call it together (each with its own triangle t of
// the same scene; t >= total_tris is an idle lane).
template <bool FILL>
__device__ __forceinline__ void bin_tri(const SceneParams& sp, int N, uint32_t t, uint32_t* count, uint32_t* cursor,
                                        uint32_t* __restrict__ list, uint32_t cap, FrameStatus* st, BinRec* big,
                                        uint32_t big_cap, uint32_t* big_count, uint32_t scene, uint2* __restrict__ rec,
                                        TriRec* __restrict__ recs) {
  const int lane = threadIdx.x & 31;
  const int nb = N / kBrick;
  float v[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
  int blo[3] = {0, 0, 0}, bhi[3] = {-1, -1, -1};
  int vol = 0;
  bool again = true;  // (filling pass) this lane's triangle is binned from scratch
  uint2 r = make_uint2(0u, 0u);
  if (FILL && t < sp.total_tris) {
    r = rec[t];
    again = (r.y & kRecAgain) != 0u;
  }
  if (again && t < sp.total_tris) {
    TriLoad tl;
    if (!FILL && recs) {
      load_tri<true>(sp, t, tl);
      if (tl.ok) store_rec(recs[t], tl);
    } else {
      load_tri<false>(sp, t, tl);
    }
    if (!tl.ok) {
      if (!FILL) atomicAdd(&st->rejected_tris, 1u);
    } else {
      const float hv = 0.5f * (float)N;
      for (int k = 0; k < 3; ++k)
        for (int d = 0; d < 3; ++d) v[k][d] = (tl.g[k][d] + 1.0f) * hv;  // voxel units
      bool inside = true;
      for (int d = 0; d < 3; ++d) {
        float lo = fminf(v[0][d], fminf(v[1][d], v[2][d])) - kBinMargin;
        float hi = fmaxf(v[0][d], fmaxf(v[1][d], v[2][d])) + kBinMargin;
        // Depth values in (-1, 0) voxel still land in voxel 0 (int() truncates).
        if (hi <= -1.0f - kBinMargin || lo >= (float)N) inside = false;
        blo[d] = max(0, (int)floorf(lo / kBrick));
        bhi[d] = min(nb - 1, (int)floorf(fmaxf(hi, 0.0f) / kBrick));
      }
      if (inside && bhi[0] >= blo[0] && bhi[1] >= blo[1] && bhi[2] >= blo[2])
        vol = (bhi[0] - blo[0] + 1) * (bhi[1] - blo[1] + 1) * (bhi[2] - blo[2] + 1);
    }
  }
  if (!FILL && vol > 0 && vol <= kSoloBricks) {
    uint32_t mask = 0u;
    int i = 0;
    for (int bz = blo[2]; bz <= bhi[2]; ++bz)
      for (int by = blo[1]; by <= bhi[1]; ++by)
        for (int bx = blo[0]; bx <= bhi[0]; ++bx, ++i)
          if (vol == 1 || touches_brick(v, bx, by, bz)) mask |= 1u << i;
    r = make_uint2((uint32_t)blo[0] | (uint32_t)blo[1] << 10 | (uint32_t)blo[2] << 20,
                   mask | (uint32_t)(bhi[0] - blo[0]) << 8 | (uint32_t)(bhi[1] - blo[1]) << 11 |
                       (uint32_t)(bhi[2] - blo[2]) << 14);
    rec[t] = r;
  }
  // The warp's triangles lie side by side, so most of its lanes meet in a brick
  // or two: one atomic for all of a brick's.  Counting and filling, us, with an
  // atomic per pair and now: 500,000 triangles 44 and 35, 37 and 18; 16 scenes
  // 251 and 148, 110 and 53.  What is left is the triangles' loads and records.
  uint32_t m = r.y & 0xffu;
  for (unsigned any = __ballot_sync(0xffffffffu, m != 0u); any; any = __ballot_sync(0xffffffffu, m != 0u)) {
    if (!m) continue;
    const int i = __ffs((int)m) - 1, ex = (int)((r.y >> 8) & 7u) + 1, ey = (int)((r.y >> 11) & 7u) + 1;
    m &= m - 1;
    const uint32_t brick = ((r.x >> 20) + (uint32_t)(i / (ex * ey))) * nb * nb +
                           (((r.x >> 10) & 1023u) + (uint32_t)((i / ex) % ey)) * nb + (r.x & 1023u) + (uint32_t)(i % ex);
    const unsigned peers = __match_any_sync(any, brick);
    const int lead = __ffs((int)peers) - 1;
    if (FILL) {
      uint32_t slot = 0;
      if (lane == lead) slot = atomicAdd(cursor + brick, (uint32_t)__popc(peers));
      slot = __shfl_sync(peers, slot, lead) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
      if (slot < cap) list[slot] = t;
    } else if (lane == lead) {
      atomicAdd(count + brick, (uint32_t)__popc(peers));
    }
  }
  bool in_warp = vol > kSoloBricks;
  if (!FILL && t < sp.total_tris && (in_warp || vol <= 0)) {
    // No bricks, or a large triangle: binned by its record (k_bin_big), or
    // where the record list is full by the warp, in both passes.  (The caller
    // is told, and may enlarge the list.)
    if (in_warp) {
      const uint32_t slot = atomicAdd(big_count, 1u);
      if (slot < big_cap) {
        in_warp = false;
        BinRec b;
        for (int k = 0; k < 3; ++k)
          for (int d = 0; d < 3; ++d) b.v[k][d] = v[k][d];
        for (int d = 0; d < 3; ++d) { b.blo[d] = blo[d]; b.bhi[d] = bhi[d]; }
        b.t = t;
        b.vol = (uint32_t)vol;
        b.scene = scene;
        b.pad = 0;
        big[slot] = b;
      }
    }
    rec[t] = make_uint2(0u, in_warp ? kRecAgain : 0u);
  }
  unsigned warp_big = __ballot_sync(0xffffffffu, in_warp);
  while (warp_big) {
    const int src = __ffs(warp_big) - 1;
    warp_big &= warp_big - 1;
    float w[3][3];
    for (int k = 0; k < 3; ++k)
      for (int d = 0; d < 3; ++d) w[k][d] = __shfl_sync(0xffffffffu, v[k][d], src);
    const int x0 = __shfl_sync(0xffffffffu, blo[0], src), y0 = __shfl_sync(0xffffffffu, blo[1], src);
    const int z0 = __shfl_sync(0xffffffffu, blo[2], src);
    const int nx = __shfl_sync(0xffffffffu, bhi[0], src) - x0 + 1;
    const int ny = __shfl_sync(0xffffffffu, bhi[1], src) - y0 + 1;
    const int n = __shfl_sync(0xffffffffu, vol, src);
    const uint32_t ts = __shfl_sync(0xffffffffu, t, src);
    for (int i = lane; i < n; i += 32)
      bin_one<FILL>(w, x0 + i % nx, y0 + (i / nx) % ny, z0 + i / (nx * ny), nb, ts, count, cursor, list, cap);
  }
}

template <bool FILL>
__global__ void __launch_bounds__(256) k_bin(SceneParams sp, int N, uint32_t* count, uint32_t* cursor,
                                             uint32_t* __restrict__ list, uint32_t cap, FrameStatus* st,
                                             BinRec* big, uint32_t big_cap, uint32_t* big_count,
                                             uint2* __restrict__ rec, TriRec* __restrict__ recs) {
  follows_previous();
  bin_tri<FILL>(sp, N, blockIdx.x * blockDim.x + threadIdx.x, count, cursor, list, cap, st, big, big_cap, big_count,
                0u, rec, recs);
}

// Every scene's triangles in one persistent launch; scene triangle ranges
// are padded to multiples of 32, so a warp bins one scene.
template <bool FILL>
__global__ void __launch_bounds__(256) k_bin_batch(BatchWork w, BatchBuffers bb) {
  follows_previous();
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < w.total; g += gridDim.x * blockDim.x) {
    const int s = batch_scene_of(w, g);
    const BatchScene& S = w.scenes[s];
    const uint32_t t = g - __ldg(w.prefix + s);
    bin_tri<FILL>(S.sp, S.N, t, FILL ? nullptr : bb.brick_count + S.brick_base,
                  FILL ? bb.brick_cursor + S.brick_base : nullptr, bb.pair_list, bb.pair_cap, bb.status, bb.big,
                  bb.big_cap, bb.big_count, (uint32_t)s,
                  bb.bin_rec + (g - t), bb.tri_rec + (g - t));
  }
}

// Large-triangle records: CTA (x, y) takes records x, x + gridDim.x, ... and
// the candidate bricks y*256 + tid, stepping by kBigSplit*256.  With
// `scenes` (a batch) each record bins into its own scene's brick slice.
template <bool FILL>
__global__ void __launch_bounds__(256) k_bin_big(int N, const BinRec* big, uint32_t big_cap,
                                                 const uint32_t* big_count, uint32_t* count, uint32_t* cursor,
                                                 uint32_t* __restrict__ list,
                                                 uint32_t cap, const BatchScene* __restrict__ scenes) {
  follows_previous();
  const uint32_t n = min(*big_count, big_cap);
  for (uint32_t r = blockIdx.x; r < n; r += gridDim.x) {
    const BinRec& rec = big[r];
    int nb = N / kBrick;
    uint32_t* cnt = count;
    uint32_t* cur = cursor;
    if (scenes) {
      const BatchScene& S = scenes[rec.scene];
      nb = S.N / kBrick;
      if (cnt) cnt += S.brick_base;
      if (cur) cur += S.brick_base;
    }
    float v[3][3];
    for (int k = 0; k < 3; ++k)
      for (int d = 0; d < 3; ++d) v[k][d] = rec.v[k][d];
    const int nx = rec.bhi[0] - rec.blo[0] + 1, ny = rec.bhi[1] - rec.blo[1] + 1;
    for (uint32_t i = blockIdx.y * blockDim.x + threadIdx.x; i < rec.vol; i += gridDim.y * blockDim.x)
      bin_one<FILL>(v, rec.blo[0] + (int)(i % nx), rec.blo[1] + (int)((i / nx) % ny), rec.blo[2] + (int)(i / (nx * ny)),
                    nb, rec.t, cnt, cur, list, cap);
  }
}

// ------------------------------------------------------------- shading -----
// voxelize.frag:124-153 in FP32.
__device__ __forceinline__ float4 voxel_color(const SceneParams& sp, const vct_material_data& m, V3 pos, V3 nrm) {
  V3 color = v3(0.f, 0.f, 0.f);
  const V3 nn = normalize(nrm);
  const int nl = min(sp.n_lights, kMaxLights);
  for (int i = 0; i < nl; ++i) {
    const vct_point_light& L = sp.lights[i];
    const V3 lp = v3(L.position[0] / sp.cube_size, L.position[1] / sp.cube_size, L.position[2] / sp.cube_size);
    const V3 dl = lp - pos;
    const V3 dir = normalize(dl);
    const float d = length(dl);
    const float a = 1.0f / (1.0f + d * d);  // attenuate(1, 0, 1, d)
    const float cs = fmaxf(dot(nn, dir), 0.0f);
    color = color + v3(L.color[0], L.color[1], L.color[2]) * (cs * a * L.intensity);
  }
  color = mulv(v3(m.diffuse[0], m.diffuse[1], m.diffuse[2]), color) + v3(m.emission[0], m.emission[1], m.emission[2]);
  float alpha = 1.0f;
  if (m.illum == 4 || m.illum == 6 || m.illum == 7 || m.illum == 9) {
    color = mulv(color, v3(m.transmittance[0], m.transmittance[1], m.transmittance[2]));
    alpha = m.dissolve;
  }
  // clamp(vec4, 0, 1) (voxelize.frag:153); with HDR storage the colour clamps to
  // [0, radiance_max] instead (radiance_max = 1 is the reference).
  const float hi = sp.radiance_max;
  return make_float4(fminf(fmaxf(color.x, 0.0f), hi), fminf(fmaxf(color.y, 0.0f), hi),
                     fminf(fmaxf(color.z, 0.0f), hi), clamp01(alpha));
}

// Per-brick sums of the contributions.  RGBA8: 16-bit fixed point per
// contribution in u32 (exact for the 1/255 result).  RGBA16F: the colour
// divided by radiance_max in 32-bit fixed point, summed in u64, so the sum
// is exact, order-independent and far finer than half precision.  Attribute
// grids (light injection): ten unorm channels in 16-bit fixed point.
template <int STORAGE> struct AccT;
// A value of the global accumulator copy, read past L1 and zeroed.
template <class T>
__device__ __forceinline__ T take_cg(T& g) {
  const T v = __ldcg(&g);
  g = 0;
  return v;
}
// v added to a 64-bit sum in shared memory, as two 32-bit atomics and a carry:
// 985 us of voxelization at 512^3, 1050 with 64-bit atomics.
__device__ __forceinline__ void add64(unsigned long long* sum, unsigned long long v) {
  uint32_t* w = reinterpret_cast<uint32_t*>(sum);
  const uint32_t lo = (uint32_t)v, old = atomicAdd(w, lo);
  const uint32_t hi = (uint32_t)(v >> 32) + (old + lo < old ? 1u : 0u);
  if (hi) atomicAdd(w + 1, hi);
}
// atomic_add_to: voxel i of these sums added into a global copy (the
// accumulator slot of a split brick); take_from: voxel i of the global copy
// read from L2 into these sums and zeroed there.
template <> struct AccT<VCT_STORAGE_RGBA8> {
  uint32_t c[4][kBrickVox];
  uint32_t n[kBrickVox];
  __device__ __forceinline__ void clear(int i) { c[0][i] = 0; c[1][i] = 0; c[2][i] = 0; c[3][i] = 0; n[i] = 0; }
  __device__ __forceinline__ void take_from(AccT& g, int i) {
    for (int k = 0; k < 4; ++k) c[k][i] = take_cg(g.c[k][i]);
    n[i] = take_cg(g.n[i]);
  }
  __device__ __forceinline__ void atomic_add_to(AccT& g, int i) const {
    if (!n[i]) return;
    for (int k = 0; k < 4; ++k)
      if (c[k][i]) atomicAdd(&g.c[k][i], c[k][i]);
    atomicAdd(&g.n[i], n[i]);
  }
  __device__ __forceinline__ void add(const SceneParams& sp, int v, const vct_material_data& m, V3 p, V3 nrm) {
    const float4 col = voxel_color(sp, m, p, nrm);
    atomicAdd(&c[0][v], __float2uint_rn(col.x * kFix));
    atomicAdd(&c[1][v], __float2uint_rn(col.y * kFix));
    atomicAdd(&c[2][v], __float2uint_rn(col.z * kFix));
    atomicAdd(&c[3][v], __float2uint_rn(col.w * kFix));
    atomicAdd(&n[v], 1u);
  }
};
template <> struct AccT<VCT_STORAGE_RGBA16F> {
  unsigned long long c[4][kBrickVox];
  uint32_t n[kBrickVox];
  __device__ __forceinline__ void clear(int i) { c[0][i] = 0; c[1][i] = 0; c[2][i] = 0; c[3][i] = 0; n[i] = 0; }
  __device__ __forceinline__ void take_from(AccT& g, int i) {
    for (int k = 0; k < 4; ++k) c[k][i] = take_cg(g.c[k][i]);
    n[i] = take_cg(g.n[i]);
  }
  __device__ __forceinline__ void atomic_add_to(AccT& g, int i) const {
    if (!n[i]) return;
    for (int k = 0; k < 4; ++k)
      if (c[k][i]) atomicAdd(&g.c[k][i], c[k][i]);
    atomicAdd(&g.n[i], n[i]);
  }
  __device__ __forceinline__ void add(const SceneParams& sp, int v, const vct_material_data& m, V3 p, V3 nrm) {
    const float4 col = voxel_color(sp, m, p, nrm);
    const float k = 4294967296.0f / sp.radiance_max;
    add64(&c[0][v], __float2ull_rn(col.x * k));
    add64(&c[1][v], __float2ull_rn(col.y * k));
    add64(&c[2][v], __float2ull_rn(col.z * k));
    add64(&c[3][v], __float2ull_rn(col.w * 4294967296.0f));
    atomicAdd(&n[v], 1u);
  }
};
// Light-injection attributes of one contribution (the factors of
// voxelize.frag:141-153 that do not depend on the lights): colour =
// t * (diffuse * lighting + emission), t = transmittance for transparent
// materials, else 1.
__device__ __forceinline__ void voxel_attrs(const vct_material_data& m, V3 nrm, float a[10]) {
  const bool tr = m.illum == 4 || m.illum == 6 || m.illum == 7 || m.illum == 9;
  const V3 t = tr ? v3(m.transmittance[0], m.transmittance[1], m.transmittance[2]) : v3(1.f, 1.f, 1.f);
  const V3 nn = normalize(nrm);
  a[0] = clamp01(m.diffuse[0] * t.x);
  a[1] = clamp01(m.diffuse[1] * t.y);
  a[2] = clamp01(m.diffuse[2] * t.z);
  a[3] = tr ? clamp01(m.dissolve) : 1.0f;
  a[4] = clamp01(0.5f * nn.x + 0.5f);
  a[5] = clamp01(0.5f * nn.y + 0.5f);
  a[6] = clamp01(0.5f * nn.z + 0.5f);
  a[7] = clamp01(m.emission[0] * t.x);
  a[8] = clamp01(m.emission[1] * t.y);
  a[9] = clamp01(m.emission[2] * t.z);
}
template <> struct AccT<kStorageAttr> {
  uint32_t c[10][kBrickVox];
  uint32_t n[kBrickVox];
  __device__ __forceinline__ void clear(int i) {
#pragma unroll
    for (int k = 0; k < 10; ++k) c[k][i] = 0;
    n[i] = 0;
  }
  __device__ __forceinline__ void take_from(AccT& g, int i) {
    for (int k = 0; k < 10; ++k) c[k][i] = take_cg(g.c[k][i]);
    n[i] = take_cg(g.n[i]);
  }
  __device__ __forceinline__ void atomic_add_to(AccT& g, int i) const {
    if (!n[i]) return;
    for (int k = 0; k < 10; ++k)
      if (c[k][i]) atomicAdd(&g.c[k][i], c[k][i]);
    atomicAdd(&g.n[i], n[i]);
  }
  __device__ __forceinline__ void add(const SceneParams&, int v, const vct_material_data& m, V3, V3 nrm) {
    float a[10];
    voxel_attrs(m, nrm, a);
#pragma unroll
    for (int k = 0; k < 10; ++k) atomicAdd(&c[k][v], __float2uint_rn(a[k] * kFix));
    atomicAdd(&n[v], 1u);
  }
};

// Mean of n 16-bit fixed-point contributions summing to c, as unorm8
// rounded to nearest (ties up): floor((510 c + 65535 n) / (2 n 65535)), both
// sides over 255; in 32 bits while n 65535 * 2 + 257 n fits.
__device__ __forceinline__ unsigned char unorm8_mean(uint32_t c, uint32_t n) {
  if (n <= 32700u && c <= n * 65535u) return (unsigned char)((2u * c + 257u * n) / (514u * n));
  const unsigned long long v = (2ull * c + 257ull * n) / (514ull * n);
  return (unsigned char)(v > 255ull ? 255ull : v);
}
typedef AccT<VCT_STORAGE_RGBA8> Acc;

// -------------------------------------------------- reference raster mode --
struct SetupRef {
  int A[3], B[3];
  float c[3];
  float farea;
  V3 gp[3], gn[3];
  uint32_t mat;
  int e[3];         // the edges at the window's first sample (row_edge)
  uint32_t window;  // first sample in the brick's columns (4 + 4 bits), samples a row - 1 (4), axis (2), fill rule (3)
};

// Returns the number of sample rows of this triangle inside the brick's columns.
template <bool REC>
__device__ int setup_ref(const SceneParams& sp, const TriRec* __restrict__ recs, int N, uint32_t t, const int b3[3], SetupRef& s) {
  TriLoad tl;
  fetch_tri<REC>(sp, recs, t, tl);
  if (!tl.ok) return 0;
  // Dominant axis, voxelize.geom:27-51 (FP32, fixed order).
  float e1[3], e2[3];
  for (int i = 0; i < 3; ++i) { e1[i] = rsub(tl.g[1][i], tl.g[0][i]); e2[i] = rsub(tl.g[2][i], tl.g[0][i]); }
  const float px = fabsf(rsub(rmul(e1[1], e2[2]), rmul(e2[1], e1[2])));
  const float py = fabsf(rsub(rmul(e1[2], e2[0]), rmul(e2[2], e1[0])));
  const float pz = fabsf(rsub(rmul(e1[0], e2[1]), rmul(e2[0], e1[1])));
  int axis;
  if (pz > px && pz > py) axis = 2;
  else if (px > py && px > pz) axis = 0;
  else axis = 1;
  const int ia = axis == 2 ? 0 : (axis == 0 ? 1 : 0);
  const int ib = axis == 2 ? 1 : 2;
  // Vertices snapped to 1/256 sample: round((g + 1) * N * 256), exactly,
  // in integer arithmetic (N is a power of two; vct_snap.h).
  const int shift = __ffs(N) - 1 + 8;
  int idx[3] = {0, 1, 2};
  long long A[3], B[3];
  float c[3];
  for (int k = 0; k < 3; ++k) {
    A[k] = snap_fixed(tl.g[k][ia], shift);
    B[k] = snap_fixed(tl.g[k][ib], shift);
    c[k] = tl.g[k][axis];
  }
  long long area = (A[1] - A[0]) * (B[2] - B[0]) - (B[1] - B[0]) * (A[2] - A[0]);
  if (area == 0) return 0;
  if (area < 0) {
    long long tA = A[1]; A[1] = A[2]; A[2] = tA;
    long long tB = B[1]; B[1] = B[2]; B[2] = tB;
    float tc = c[1]; c[1] = c[2]; c[2] = tc;
    idx[1] = 2; idx[2] = 1;
    area = -area;
  }
  // Sample window: the triangle's sample bbox inside the brick's columns.
  const long long minA = min(A[0], min(A[1], A[2])), maxA = max(A[0], max(A[1], A[2]));
  const long long minB = min(B[0], min(B[1], B[2])), maxB = max(B[0], max(B[1], B[2]));
  const int sa0 = 2 * kBrick * b3[ia], sb0 = 2 * kBrick * b3[ib];
  const long long i0 = max((long long)sa0, ceil_div(minA - 128, 256));
  const long long i1 = min((long long)sa0 + 2 * kBrick - 1, floor_div(maxA - 128, 256));
  const long long j0 = max((long long)sb0, ceil_div(minB - 128, 256));
  const long long j1 = min((long long)sb0 + 2 * kBrick - 1, floor_div(maxB - 128, 256));
  if (i1 < i0 || j1 < j0) return 0;
  s.farea = __ll2float_rn(area);
  for (int k = 0; k < 3; ++k) {
    s.A[k] = (int)A[k];
    s.B[k] = (int)B[k];
    s.c[k] = c[k];
    const int o = idx[k];
    s.gp[k] = v3(tl.g[o][0], tl.g[o][1], tl.g[o][2]);
    s.gn[k] = tl.n[o];
  }
  for (int k = 0; k < 3; ++k) {
    const int a = (k + 1) % 3, b = (k + 2) % 3;
    s.e[k] = row_edge(A[a], B[a], A[b], B[b], top_left(A[a], B[a], A[b], B[b]), (int)i0, (int)j0);
  }
  s.mat = tl.mat;
  s.window = (uint32_t)(i0 - sa0) | (uint32_t)(j0 - sb0) << 4 | (uint32_t)(i1 - i0) << 8 | (uint32_t)axis << 12;
  return (int)(j1 - j0 + 1);
}

// The covered samples of row `row` of the setup's window, as bits; `code` +
// their index: the sample in the brick's columns, i in the low 4 bits.
__device__ __forceinline__ uint32_t cover(const SetupRef& s, int row, uint32_t& code) {
  const uint32_t w = s.window;
  code = (w & 15u) | ((w >> 4 & 15u) + (uint32_t)row) << 4;
  int e[3], ey[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int a = (k + 1) % 3, b = (k + 2) % 3;
    e[k] = s.e[k] + (s.A[b] - s.A[a]) * row;
    ey[k] = s.B[b] - s.B[a];
  }
  return row_mask(e[0], e[1], e[2], ey[0], ey[1], ey[2], (int)(w >> 8 & 15u) + 1);
}

// One covered sample.
template <class A>
__device__ __forceinline__ void hit(const SceneParams& sp, int N, const int b3[3], const SetupRef& s, uint32_t code,
                                    A& acc) {
  const int axis = (int)(s.window >> 12 & 3u);
  const int i = 2 * kBrick * (axis == 0 ? b3[1] : b3[0]) + (int)(code & 15u);
  const int j = 2 * kBrick * (axis == 2 ? b3[1] : b3[2]) + (int)(code >> 4 & 15u);
  const long long sx = 256LL * i + 128, sy = 256LL * j + 128;
  const long long w0 = edge_fn(s.A[1], s.B[1], s.A[2], s.B[2], sx, sy);
  const long long w1 = edge_fn(s.A[2], s.B[2], s.A[0], s.B[0], sx, sy);
  const long long w2 = edge_fn(s.A[0], s.B[0], s.A[1], s.B[1], sx, sy);
  const float b1 = rdiv(__ll2float_rn(w1), s.farea), b2 = rdiv(__ll2float_rn(w2), s.farea);
  float cz = radd(s.c[0], rmul(b1, rsub(s.c[1], s.c[0])));
  cz = radd(cz, rmul(b2, rsub(s.c[2], s.c[0])));
  const float Nf = (float)N;
  const float t = rmul(Nf, radd(rmul(0.5f, cz), 0.5f));
  if (!(t > -1.0f && t < Nf)) return;
  const int kd = __float2int_rz(t);
  int vx, vy, vz;
  if (axis == 2) { vx = i >> 1; vy = j >> 1; vz = kd; }
  else if (axis == 0) { vx = kd; vy = i >> 1; vz = j >> 1; }
  else { vx = i >> 1; vy = kd; vz = j >> 1; }
  const int lx = vx - b3[0] * kBrick, ly = vy - b3[1] * kBrick, lz = vz - b3[2] * kBrick;
  if ((unsigned)lx >= (unsigned)kBrick || (unsigned)ly >= (unsigned)kBrick || (unsigned)lz >= (unsigned)kBrick) return;
  const float l0 = __ll2float_rn(w0) / s.farea, l1 = __ll2float_rn(w1) / s.farea, l2 = __ll2float_rn(w2) / s.farea;
  const V3 p = s.gp[0] * l0 + s.gp[1] * l1 + s.gp[2] * l2;
  const V3 n = s.gn[0] * l0 + s.gn[1] * l1 + s.gn[2] * l2;
  acc.add(sp, (lz * kBrick + ly) * kBrick + lx, sp.materials[s.mat], p, n);
}

// ---------------------------------------------------- conservative mode ----
struct SetupSat {
  int V[3][3];  // relative to the brick
  V3 gp[3], gn[3];
  uint32_t mat;
  // The triangle's box in the brick: first voxel (3 x 3 bits), voxels - 1
  // across x (3) and down z (3), ceil(512 / voxels across x) (10), the form
  // of the test (2).
  uint32_t box;
};

// Returns the number of columns (along z) of the triangle's box in the brick.
template <bool REC>
__device__ int setup_sat(const SceneParams& sp, const TriRec* __restrict__ recs, int N, uint32_t t, const int b3[3], SetupSat& s) {
  TriLoad tl;
  fetch_tri<REC>(sp, recs, t, tl);
  if (!tl.ok) return 0;
  // Vertices snapped to 1/256 voxel: round((g + 1) * N * 128), exactly, in
  // integer arithmetic (N is a power of two; vct_snap.h).
  const int shift = __ffs(N) - 1 + 7;
  int lo[3], hi[3];
  long long extent = 0;
  for (int d = 0; d < 3; ++d) {
    const int origin = b3[d] * kBrick * 256;
    int mn = INT_MAX, mx = INT_MIN;
    for (int k = 0; k < 3; ++k) {
      const int q = (int)snap_fixed(tl.g[k][d], shift) - origin;
      s.V[k][d] = q;
      mn = min(mn, q);
      mx = max(mx, q);
    }
    extent = max(extent, (long long)mx - mn);
    lo[d] = max(0, ((mn + 255) >> 8) - 1);
    hi[d] = min(kBrick - 1, mx >> 8);
    if (hi[d] < lo[d]) return 0;
  }
  for (int k = 0; k < 3; ++k) {
    s.gp[k] = v3(tl.g[k][0], tl.g[k][1], tl.g[k][2]);
    s.gn[k] = tl.n[k];
  }
  s.mat = tl.mat;
  const uint32_t nx = (uint32_t)(hi[0] - lo[0] + 1), form = extent <= kSatInt ? 0u : extent <= kSatLong ? 1u : 2u;
  s.box = (uint32_t)lo[0] | (uint32_t)lo[1] << 3 | (uint32_t)lo[2] << 6 | (nx - 1) << 9 |
          (uint32_t)(hi[2] - lo[2]) << 12 | ((511u + nx) / nx) << 15 | form << 25;
  return (int)nx * (hi[1] - lo[1] + 1);
}

// The column test's forms for triangles that are large beside a brick, called
// so that the kernel's body holds the 32-bit form alone.
__device__ __noinline__ uint32_t cover_large(const SetupSat& s, bool wide, int x, int y, int z0, int nz) {
  if (wide) return sat_column<long long>(s.V, x, y, z0, nz);
  uint32_t mask = 0;
#pragma unroll 1
  for (int k = 0; k < nz; ++k) mask |= (sat_exact(s.V, x, y, z0 + k) ? 1u : 0u) << k;
  return mask;
}

// The touched voxels of column `col` of the setup's box, as bits; `code` +
// their index: the voxel in the brick, z in the low 3 bits.
__device__ __forceinline__ uint32_t cover(const SetupSat& s, int col, uint32_t& code) {
  const uint32_t w = s.box;
  const int nx = (int)(w >> 9 & 7u) + 1, nz = (int)(w >> 12 & 7u) + 1;
  const int row = (int)((uint32_t)col * (w >> 15 & 1023u) >> 9);  // col / nx: col < 64, so exact
  const int x = (int)(w & 7u) + col - row * nx, y = (int)(w >> 3 & 7u) + row, z0 = (int)(w >> 6 & 7u);
  code = (uint32_t)(z0 | y << 3 | x << 6);
  const uint32_t form = w >> 25;
  if (form == 0u) return sat_column<int>(s.V, x, y, z0, nz);
  return cover_large(s, form == 1u, x, y, z0, nz);
}

// Barycentric weights of the closest triangle point to p (Voronoi-region
// classification of vertices, edges and face).
__device__ void closest_bary(V3 p, V3 a, V3 b, V3 c, float w[3]) {
  const V3 ab = b - a, ac = c - a, ap = p - a;
  const float d1 = dot(ab, ap), d2 = dot(ac, ap);
  if (d1 <= 0.f && d2 <= 0.f) { w[0] = 1.f; w[1] = 0.f; w[2] = 0.f; return; }
  const V3 bp = p - b;
  const float d3 = dot(ab, bp), d4 = dot(ac, bp);
  if (d3 >= 0.f && d4 <= d3) { w[0] = 0.f; w[1] = 1.f; w[2] = 0.f; return; }
  const float vc = d1 * d4 - d3 * d2;
  if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
    const float den = d1 - d3, v = den != 0.f ? d1 / den : 0.f;
    w[0] = 1.f - v; w[1] = v; w[2] = 0.f; return;
  }
  const V3 cp = p - c;
  const float d5 = dot(ab, cp), d6 = dot(ac, cp);
  if (d6 >= 0.f && d5 <= d6) { w[0] = 0.f; w[1] = 0.f; w[2] = 1.f; return; }
  const float vb = d5 * d2 - d1 * d6;
  if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
    const float den = d2 - d6, t = den != 0.f ? d2 / den : 0.f;
    w[0] = 1.f - t; w[1] = 0.f; w[2] = t; return;
  }
  const float va = d3 * d6 - d5 * d4;
  if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
    const float den = (d4 - d3) + (d5 - d6), t = den != 0.f ? (d4 - d3) / den : 0.f;
    w[0] = 0.f; w[1] = 1.f - t; w[2] = t; return;
  }
  const float sum = va + vb + vc;
  if (!(sum != 0.f)) { w[0] = 1.f; w[1] = 0.f; w[2] = 0.f; return; }
  const float v = vb / sum, t = vc / sum;
  w[0] = 1.f - v - t; w[1] = v; w[2] = t;
}

// One touched voxel.
template <class A>
__device__ __forceinline__ void hit(const SceneParams& sp, int N, const int b3[3], const SetupSat& s, uint32_t code,
                                    A& acc) {
  const int lx = (int)(code >> 6 & 7u), ly = (int)(code >> 3 & 7u), lz = (int)(code & 7u);
  const int x = b3[0] * kBrick + lx, y = b3[1] * kBrick + ly, z = b3[2] * kBrick + lz;
  const float inv = 2.0f / (float)N;
  const V3 vc = v3(((float)x + 0.5f) * inv - 1.0f, ((float)y + 0.5f) * inv - 1.0f, ((float)z + 0.5f) * inv - 1.0f);
  float w[3];
  closest_bary(vc, s.gp[0], s.gp[1], s.gp[2], w);
  const V3 p = s.gp[0] * w[0] + s.gp[1] * w[1] + s.gp[2] * w[2];
  const V3 n = s.gn[0] * w[0] + s.gn[1] * w[1] + s.gn[2] * w[2];
  acc.add(sp, (lz * kBrick + ly) * kBrick + lx, sp.materials[s.mat], p, n);
}

// ------------------------------------------------------------ brick CTA ----
template <int MODE>
using SetupOf = typename std::conditional<MODE == VCT_VOX_CONSERVATIVE, SetupSat, SetupRef>::type;

// Shared memory of a round of pairs.
template <int MODE>
struct RoundOf {
  SetupOf<MODE> setup[kRound];
  int first[kRound];           // a pair's first row (column) among the round's
  uint16_t queue[kWarps][64];  // covered samples not yet shaded: pair << 9 | code
  int sum[kWarps];
};
static_assert(kRound <= 128, "a queue entry holds the pair in 7 bits");

// Accumulates the (triangle, brick) pairs list[beg, end) of the brick at b3
// into acc (all threads of the CTA; cleared first, barrier at the end).
// Rounds of up to kRound pairs: a setup per thread, a scan of the pairs' rows
// (columns), then every warp tests rows in turn, a lane each, and queues what
// is covered; it shades a full warp's worth from the queue at a time: of the
// samples tested a third to a half are covered, and shading one costs ten
// times the test.  (64-bit tests, each followed at once by its shading, and a
// CTA per brick of the grid, 512^3 and two million triangles, conservative:
// 1423 us, 256^3 and 500,000, raster: 215; now 737 and 150.  Half of that is
// the pairs' loads and setup, a quarter shading.)
template <int MODE, int STORAGE, bool REC>
__device__ __forceinline__ void brick_accumulate(const SceneParams& sp, const TriRec* __restrict__ recs, int N, const int b3[3],
                                                 const uint32_t* list, uint32_t beg, uint32_t end,
                                                 AccT<STORAGE>& acc, RoundOf<MODE>& rd) {
  for (int i = threadIdx.x; i < kBrickVox; i += kThreads) acc.clear(i);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint16_t* queue = rd.queue[warp];
  for (uint32_t b0 = beg; b0 < end; b0 += kRound) {
    const uint32_t n = min((uint32_t)kRound, end - b0);
    int cnt = 0;
    if ((uint32_t)threadIdx.x < n) {
      const uint32_t t = list[b0 + threadIdx.x];
      if constexpr (MODE == VCT_VOX_CONSERVATIVE) cnt = setup_sat<REC>(sp, recs, N, t, b3, rd.setup[threadIdx.x]);
      else cnt = setup_ref<REC>(sp, recs, N, t, b3, rd.setup[threadIdx.x]);
    }
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) rd.sum[warp] = incl;
    __syncthreads();
    int off = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int v = rd.sum[w];
      off += w < warp ? v : 0;
      total += v;
    }
    if (threadIdx.x < kRound) rd.first[threadIdx.x] = off + incl - cnt;
    __syncthreads();
    int at = 0, queued = 0;
    uint32_t mask = 0, code = 0;
    for (;;) {
      while (queued < 32) {
        const unsigned some = __ballot_sync(0xffffffffu, mask != 0u);
        if (some) {  // one covered sample of every lane that has any
          if (mask) {
            queue[queued + __popc(some & ((1u << lane) - 1u))] = (uint16_t)(code + (uint32_t)__ffs((int)mask) - 1u);
            mask &= mask - 1u;
          }
          queued += __popc(some);
          continue;
        }
        if (at >= total) break;
        const int it = at + lane * kWarps + warp;  // (a few rows reach every warp)
        at += kThreads;
        if (it < total) {
          int lo = 0, hi = (int)n - 1;  // owner = last pair with first <= it
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (rd.first[mid] <= it) lo = mid; else hi = mid - 1;
          }
          mask = cover(rd.setup[lo], it - rd.first[lo], code);
          code |= (uint32_t)lo << 9;
        }
      }
      const int m = min(queued, 32);
      if (m == 0) break;
      __syncwarp();
      queued -= m;
      if (lane < m) {
        const uint32_t q = queue[queued + lane];
        hit(sp, N, b3, rd.setup[q >> 9], q & 511u, acc);
      }
      __syncwarp();  // the entries are read before their place is written again
    }
    __syncthreads();  // the round's setups and offsets are free again
  }
}

// ---- fused mip levels 1-3 (six maps, RGBA8 or RGBA16F; BrickMips) ---------
// The brick holds whole 4^3, 2^3 and 1^3 blocks of levels 1-3, so its CTA
// writes them from its level-0 texels in shared memory with the MipBuilder's
// rule (vct_mip.cuh: exact integers for RGBA8, one fixed FP32 evaluation for
// RGBA16F), plus the alpha chains and the occupancy bytes of
// those levels (a cell is occupied when its block of level 0 holds a
// non-zero texel); the MipBuilder then starts from level 3.  This replaces
// the first pass's re-read of level 0 (and the linear copy it read).
template <int STORAGE>
struct BrickMipScratchT {
  typedef typename std::conditional<STORAGE == VCT_STORAGE_RGBA16F, uint2, uint32_t>::type T;
  T l0[kBrick * kBrick * kBrick];
  T l1[6][64];
  T l2[6][8];
  T l3[6];
  uint8_t occ1[64];
  uint8_t occ2[8];
};
typedef BrickMipScratchT<VCT_STORAGE_RGBA8> BrickMipScratch;
__device__ __forceinline__ bool texel_nonzero(uint32_t v) { return v != 0u; }
__device__ __forceinline__ bool texel_nonzero(uint2 v) { return (v.x | v.y) != 0u; }

template <class T>
__device__ __forceinline__ void brick_alpha(const BrickMips& bm, int level, int x, int y, int z, const T* v,
                                            int stride) {
#pragma unroll
  for (int c = 0; c < kMaxAlpha; ++c)
    surf3Dwrite(alpha_texel(v, stride, c), bm.alpha[c][level], x * (int)sizeof(T), y, z);
}

__device__ __forceinline__ void brick_occ(const BrickMips& bm, int N, int level, int x, int y, int z, bool any) {
  if (!bm.occ_raw[level]) return;
  const int s = N >> level;
  bm.occ_raw[level][((size_t)z * s + y) * s + x] = any ? 1 : 0;
}

// Texel (x, y, z), map d, of the level above a cube of side s2 stored
// [z][y][x] at src (shared memory): one out-of-line copy of the rule for
// all three levels.
__device__ __noinline__ uint32_t brick_mip_texel(const uint32_t* src, int s2, int x, int y, int z, int d) {
  return aniso_rgba8_dir(d, [&](int k) { return src[mip_child(s2, x, y, z, k)]; });
}
__device__ __noinline__ uint2 brick_mip_texel(const uint2* src, int s2, int x, int y, int z, int d) {
  return aniso_rgba16f_dir(d, [&](int k) { return src[mip_child(s2, x, y, z, k)]; });
}

// Levels 1-3 of brick b3 from scr.l0 ([z][y][x], written and synchronised
// by the caller); all threads of the CTA.  Level 1 takes the whole CTA, one
// (texel, map) item per thread with the map a run-time index, so that the
// rule's code exists once (six unrolled copies made the kernel miss its
// instruction cache); levels 2 and 3 (48 and 6 items) and their occupancy
// and alpha copies are one warp's, which synchronises only itself.
template <int STORAGE>
__device__ void brick_mips(const BrickMips& bm, int N, const int b3[3], BrickMipScratchT<STORAGE>& scr) {
  static_assert(kThreads >= 96, "levels 2-3 are warp 2's");
  typedef typename BrickMipScratchT<STORAGE>::T T;
  constexpr int kB = sizeof(T);  // bytes per texel
  const int t = threadIdx.x;
  for (int i = t; i < 6 * 64; i += kThreads) {  // level 1: map i / 64 (warp-uniform), texel i % 64
    const int d = i >> 6, r = i & 63, x = r & 3, y = (r >> 2) & 3, z = r >> 4;
    const T v = brick_mip_texel(scr.l0, 8, x, y, z, d);
    surf3Dwrite(v, bm.surf[d][1], (b3[0] * 4 + x) * kB, b3[1] * 4 + y, b3[2] * 4 + z);
    scr.l1[d][r] = v;
  }
  if (t < 64) {  // occupancy of level 1: the texel's block of level 0
    const int x = t & 3, y = (t >> 2) & 3, z = t >> 4;
    bool any = false;
#pragma unroll
    for (int k = 0; k < 8; ++k) any |= texel_nonzero(scr.l0[mip_child(8, x, y, z, k)]);
    scr.occ1[t] = any ? 1 : 0;
    brick_occ(bm, N, 1, b3[0] * 4 + x, b3[1] * 4 + y, b3[2] * 4 + z, any);
  }
  __syncthreads();
  if (t < 64) {
    if (bm.has_alpha) brick_alpha(bm, 1, b3[0] * 4 + (t & 3), b3[1] * 4 + ((t >> 2) & 3), b3[2] * 4 + (t >> 4),
                                  &scr.l1[0][t], 64);
    return;
  }
  if (t >= 96) return;
  const int lane = t - 64;
  for (int j = lane; j < 48; j += 32) {  // level 2: texel r of map d from that map's level 1
    const int d = j >> 3, r = j & 7, x = r & 1, y = (r >> 1) & 1, z = r >> 2;
    const T v = brick_mip_texel(scr.l1[d], 4, x, y, z, d);
    surf3Dwrite(v, bm.surf[d][2], (b3[0] * 2 + x) * kB, b3[1] * 2 + y, b3[2] * 2 + z);
    scr.l2[d][r] = v;
  }
  if (lane < 8) {  // occupancy of level 2 from level 1's
    const int x = lane & 1, y = (lane >> 1) & 1, z = lane >> 2;
    bool any = false;
#pragma unroll
    for (int k = 0; k < 8; ++k) any |= scr.occ1[mip_child(4, x, y, z, k)] != 0;
    scr.occ2[lane] = any ? 1 : 0;
    brick_occ(bm, N, 2, b3[0] * 2 + x, b3[1] * 2 + y, b3[2] * 2 + z, any);
  }
  __syncwarp();
  if (lane < 8) {
    if (bm.has_alpha)
      brick_alpha(bm, 2, b3[0] * 2 + (lane & 1), b3[1] * 2 + ((lane >> 1) & 1), b3[2] * 2 + (lane >> 2),
                  &scr.l2[0][lane], 8);
  } else if (lane < 14) {  // level 3: the brick's one texel of map d
    const int d = lane - 8;
    const T v = brick_mip_texel(scr.l2[d], 2, 0, 0, 0, d);
    surf3Dwrite(v, bm.surf[d][3], b3[0] * kB, b3[1], b3[2]);
    scr.l3[d] = v;
  } else if (lane == 14) {
    bool any = false;
    for (int k = 0; k < 8; ++k) any |= scr.occ2[k] != 0;
    brick_occ(bm, N, 3, b3[0], b3[1], b3[2], any);
  }
  __syncwarp();
  if (lane == 0 && bm.has_alpha) brick_alpha(bm, 3, b3[0], b3[1], b3[2], scr.l3, 1);
}

// Levels 1-3 of an empty brick: zeros (the texels and the occupancy).
template <int STORAGE>
__device__ void brick_mips_zero(const BrickMips& bm, int N, const int b3[3]) {
  const int t = threadIdx.x;
  const typename BrickMipScratchT<STORAGE>::T zero[6] = {};
  int level = 0, x = 0, y = 0, z = 0;
  if (t < 64) {
    level = 1;
    x = b3[0] * 4 + (t & 3);
    y = b3[1] * 4 + ((t >> 2) & 3);
    z = b3[2] * 4 + (t >> 4);
  } else if (t < 72) {
    level = 2;
    x = b3[0] * 2 + (t & 1);
    y = b3[1] * 2 + ((t >> 1) & 1);
    z = b3[2] * 2 + ((t >> 2) & 1);
  } else if (t == 72) {
    level = 3;
    x = b3[0];
    y = b3[1];
    z = b3[2];
  }
  if (!level) return;
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    if constexpr (STORAGE == VCT_STORAGE_RGBA16F) surf3Dwrite(make_uint2(0u, 0u), bm.surf[d][level], x * 8, y, z);
    else surf3Dwrite(0u, bm.surf[d][level], x * 4, y, z);
  }
  if (bm.has_alpha) brick_alpha(bm, level, x, y, z, zero, 1);
  brick_occ(bm, N, level, x, y, z, false);
}

// Writes the brick at b3 from its sums: order-independent mean, round to
// nearest (ties up); empty voxels = 0.  `acc` may be in shared or global
// memory.
// SURF: level 0 through the surface (else into l0_lin alone).
template <int STORAGE, bool SURF = true>
__device__ __forceinline__ void brick_finalize(const SceneParams& sp, int N, const int b3[3], const AccT<STORAGE>& acc,
                                               cudaSurfaceObject_t l0, uint32_t* __restrict__ counts,
                                               FrameStatus* st, const InjGrids& inj, void* l0_lin,
                                               const BrickMips* bm = nullptr, void* scr_raw = nullptr) {
  using Scr = BrickMipScratchT<STORAGE == VCT_STORAGE_RGBA16F ? VCT_STORAGE_RGBA16F : VCT_STORAGE_RGBA8>;
  Scr* scr = static_cast<Scr*>(scr_raw);
  for (int i = threadIdx.x; i < kBrickVox; i += kThreads) {
    const uint32_t n = acc.n[i];
    const int lx = i & 7, ly = (i >> 3) & 7, lz = i >> 6;
    const int x = b3[0] * kBrick + lx, y = b3[1] * kBrick + ly, z = b3[2] * kBrick + lz;
    if (n > 65535u) atomicAdd(&st->count_saturated, 1u);
    if constexpr (STORAGE == kStorageAttr) {
      uchar4 a = make_uchar4(0, 0, 0, 0), nn = a, e = a;
      if (n) {
        a = make_uchar4(unorm8_mean(acc.c[0][i], n), unorm8_mean(acc.c[1][i], n), unorm8_mean(acc.c[2][i], n),
                        unorm8_mean(acc.c[3][i], n));
        nn = make_uchar4(unorm8_mean(acc.c[4][i], n), unorm8_mean(acc.c[5][i], n), unorm8_mean(acc.c[6][i], n), 0);
        e = make_uchar4(unorm8_mean(acc.c[7][i], n), unorm8_mean(acc.c[8][i], n), unorm8_mean(acc.c[9][i], n), 255);
      }
      surf3Dwrite(a, inj.albedo, x * 4, y, z);
      surf3Dwrite(nn, inj.normal, x * 4, y, z);
      surf3Dwrite(e, inj.emission, x * 4, y, z);
    } else if constexpr (STORAGE == VCT_STORAGE_RGBA8) {
      uchar4 o = make_uchar4(0, 0, 0, 0);
      if (n) o = make_uchar4(unorm8_mean(acc.c[0][i], n), unorm8_mean(acc.c[1][i], n), unorm8_mean(acc.c[2][i], n),
                             unorm8_mean(acc.c[3][i], n));
      if constexpr (SURF) surf3Dwrite(o, l0, x * 4, y, z);
      if (l0_lin) static_cast<uchar4*>(l0_lin)[((size_t)z * N + y) * N + x] = o;
      if (bm) scr->l0[i] = (uint32_t)o.x | (uint32_t)o.y << 8 | (uint32_t)o.z << 16 | (uint32_t)o.w << 24;
    } else {
      ushort4 o = make_ushort4(0, 0, 0, 0);
      if (n) {
        const float inv = 1.0f / ((float)n * 4294967296.0f), k = inv * sp.radiance_max;
        o = make_ushort4(__half_as_ushort(__float2half_rn((float)acc.c[0][i] * k)),
                         __half_as_ushort(__float2half_rn((float)acc.c[1][i] * k)),
                         __half_as_ushort(__float2half_rn((float)acc.c[2][i] * k)),
                         __half_as_ushort(__float2half_rn((float)acc.c[3][i] * inv)));
      }
      surf3Dwrite(o, l0, x * 8, y, z);
      if (l0_lin) static_cast<ushort4*>(l0_lin)[((size_t)z * N + y) * N + x] = o;
      if (bm) scr->l0[i] = make_uint2((uint32_t)o.x | (uint32_t)o.y << 16, (uint32_t)o.z | (uint32_t)o.w << 16);
    }
    if (counts) counts[((size_t)z * N + y) * N + x] = n;
  }
  if constexpr (STORAGE == VCT_STORAGE_RGBA8 || STORAGE == VCT_STORAGE_RGBA16F) {
    if (bm) {
      __syncthreads();
      brick_mips<STORAGE>(*bm, N, b3, *scr);
    }
  }
}

__device__ __forceinline__ void brick_coords(int N, uint32_t brick, int b3[3]) {
  const int nb = N / kBrick;
  b3[0] = (int)(brick % nb);
  b3[1] = (int)((brick / nb) % nb);
  b3[2] = (int)(brick / ((uint32_t)nb * nb));
}

// One unit of brick work, all threads of the CTA (the shared-memory arrays
// come from the caller, so that a persistent CTA reuses them unit after
// unit): the whole brick, or -- for a dense brick with an accumulator slot
// (hb->slot[slot_index] >= 0) -- its chunk `chunk`.
// A chunk adds its sums into the slot; the CTA that completes the brick's
// last chunk takes the sums back (zeroing the slot and its counter for the
// next frame) and writes the brick.  `item`: the unit is an extra chunk
// (>= 1) of a split brick.  Every kernel calls this from one place only,
// so that its code exists once per kernel (instruction-cache footprint).
template <int MODE, int STORAGE, bool SURF = true, bool REC = true>
__device__ __forceinline__ void brick_unit(const SceneParams& sp, const TriRec* __restrict__ recs, int N, uint32_t brick,
                                           const uint32_t* offset, const uint32_t* list,
                                           uint32_t cap, cudaSurfaceObject_t l0, uint32_t* __restrict__ counts,
                                           FrameStatus* st, AccT<STORAGE>& acc, RoundOf<MODE>& rd, const InjGrids& inj, void* l0_lin,
                                           const HeavyBricks* hb, uint32_t slot_index, uint32_t chunk, bool item,
                                           const BrickMips* bm = nullptr, uint8_t* dirty = nullptr) {
  static_assert(sizeof(BrickMipScratchT<VCT_STORAGE_RGBA16F>) <= sizeof(rd),
                "fused mips fit in the round's memory");
  __shared__ uint32_t s_last;
  int b3[3];
  brick_coords(N, brick, b3);
  const uint32_t beg0 = min(offset[brick], cap), end = min(offset[brick + 1], cap);
  if (beg0 == end) {
    // No triangle touches this brick (most of the grid): store cleared texels
    // without the accumulator or its barriers -- unless they are zero already
    // (`dirty`: per brick, 1 when its texels -- level 0, its linear copy and
    // any fused levels -- may be non-zero; the per-voxel counts are not
    // tracked by it).
    if (dirty && !counts) {
      if (!dirty[brick]) return;  // CTA-uniform
      __syncthreads();            // every thread has read the flag
      if (threadIdx.x == 0) dirty[brick] = 0;
    }
    for (int i = threadIdx.x; i < kBrickVox; i += kThreads) {
      const int x = b3[0] * kBrick + (i & 7), y = b3[1] * kBrick + ((i >> 3) & 7), z = b3[2] * kBrick + (i >> 6);
      if (STORAGE == kStorageAttr) {
        surf3Dwrite(make_uchar4(0, 0, 0, 0), inj.albedo, x * 4, y, z);
        surf3Dwrite(make_uchar4(0, 0, 0, 0), inj.normal, x * 4, y, z);
        surf3Dwrite(make_uchar4(0, 0, 0, 0), inj.emission, x * 4, y, z);
      } else if (STORAGE == VCT_STORAGE_RGBA8) {
        if constexpr (SURF) surf3Dwrite(make_uchar4(0, 0, 0, 0), l0, x * 4, y, z);
        if (l0_lin) static_cast<uchar4*>(l0_lin)[((size_t)z * N + y) * N + x] = make_uchar4(0, 0, 0, 0);
      } else {
        surf3Dwrite(make_ushort4(0, 0, 0, 0), l0, x * 8, y, z);
        if (l0_lin) static_cast<ushort4*>(l0_lin)[((size_t)z * N + y) * N + x] = make_ushort4(0, 0, 0, 0);
      }
      if (counts) counts[((size_t)z * N + y) * N + x] = 0u;
    }
    if constexpr (STORAGE == VCT_STORAGE_RGBA8 || STORAGE == VCT_STORAGE_RGBA16F)
      if (bm) brick_mips_zero<STORAGE>(*bm, N, b3);
    return;
  }
  // Only a dense brick looks up its slot.
  const int slot = (hb && hb->slot && (item || end - beg0 > kHeavyChunk)) ? hb->slot[slot_index] : -1;
  uint32_t beg = beg0, stop = end;
  if (slot >= 0) {
    const uint32_t span = heavy_span(end - beg0);
    beg = min(beg0 + chunk * span, end);
    stop = min(beg + span, end);
  }
  brick_accumulate<MODE, STORAGE, REC>(sp, recs, N, b3, list, beg, stop, acc, rd);
  if (slot >= 0) {
    AccT<STORAGE>& g = static_cast<AccT<STORAGE>*>(hb->acc)[slot];
    for (int i = threadIdx.x; i < kBrickVox; i += kThreads) acc.atomic_add_to(g, i);
    __threadfence();  // this CTA's sums are in L2 before its chunk counts as done
    __syncthreads();
    if (threadIdx.x == 0) {
      const uint32_t nch = heavy_chunks(end - beg0);
      s_last = atomicAdd(&hb->done[slot], 1u) == nch - 1 ? 1u : 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int i = threadIdx.x; i < kBrickVox; i += kThreads) acc.take_from(g, i);
    if (threadIdx.x == 0) hb->done[slot] = 0;
    __syncthreads();
  }
  // (the round is done with: its memory holds the fused mips)
  if (dirty && threadIdx.x == 0) dirty[brick] = 1;
  brick_finalize<STORAGE, SURF>(sp, N, b3, acc, l0, counts, st, inj, l0_lin, bm, &rd);
}

// The list of bricks with work in `words` (4 + bricks words).
BrickUnits brick_units(uint32_t* words, uint32_t bricks, const uint8_t* dirty, uint32_t* reset) {
  BrickUnits u;
  u.list = words + 4;
  u.count = words;
  u.cap = bricks;
  u.dirty = dirty;
  u.reset = reset;
  return u;
}

// Runs f(brick, chunk, extra) for the units this CTA takes: one by its index,
// then from the counter, fetched while the unit before it runs.  The extra
// chunks of the split bricks come first, so that they do not end the launch,
// then the long bricks, then the others.  (A CTA per brick of the grid spent
// 512^3 voxelization 280 us on the empty ones, seven in eight.)
template <class F>
__device__ __forceinline__ void for_units(const HeavyBricks& hb, const BrickUnits& u, FrameStatus* st, F&& f) {
  __shared__ uint32_t s_next[2];
  follows_previous();
  if (u.reset && blockIdx.x == 0 && threadIdx.x == 0) *u.reset = 0u;
  const uint32_t n_items = hb.slot ? min(hb.counters[1], hb.item_cap) : 0u, n_long = u.count[0];
  const uint32_t total = n_items + n_long + u.count[1];
  if (hb.slot && blockIdx.x == 0 && threadIdx.x < 2) (&st->heavy_total)[threadIdx.x] = hb.counters[threadIdx.x];
  int turn = 0;
  for (uint32_t q = blockIdx.x; q < total; turn ^= 1) {
    if (threadIdx.x == 0) s_next[turn] = gridDim.x + atomicAdd(&u.count[2], 1u);
    const uint32_t i = q - n_items;
    const bool extra = q < n_items;
    const uint2 w = extra ? hb.items[q] : make_uint2(u.list[i < n_long ? i : u.cap - 1u - (i - n_long)], 0u);
    if (w.x != 0xffffffffu) f(w.x, w.y, extra);  // (an unused item: CTA-uniform)
    __syncthreads();  // the unit is done with its shared memory
    q = s_next[turn];
  }
}

// (FUSE: with the fused mips.)
template <int MODE, int STORAGE, bool FUSE = false>
__global__ void __launch_bounds__(kThreads, brick_min_blocks<STORAGE>()) k_bricks(SceneParams sp, int N, const uint32_t* offset,
                                                     const uint32_t* list, uint32_t cap,
                                                     cudaSurfaceObject_t l0, uint32_t* __restrict__ counts,
                                                     FrameStatus* st, InjGrids inj, void* l0_lin, HeavyBricks hb,
                                                     BrickUnits units, const TriRec* __restrict__ recs,
                                                     const __grid_constant__ BrickMips bm) {
  __shared__ AccT<STORAGE> acc;
  __shared__ __align__(8) RoundOf<MODE> rd;
  for_units(hb, units, st, [&](uint32_t brick, uint32_t chunk, bool extra) {
    brick_unit<MODE, STORAGE>(sp, recs, N, brick, offset, list, cap, l0, counts, st, acc, rd, inj, l0_lin, &hb, brick, chunk,
                              extra, FUSE ? &bm : nullptr, bm.dirty);
  });
}

// Every scene's bricks in one launch.
template <int MODE, int STORAGE, bool FUSE = false>
__global__ void __launch_bounds__(kThreads, brick_min_blocks<STORAGE>())
    k_bricks_batch(BatchWork w, BatchBuffers bb, BrickUnits units) {
  __shared__ AccT<STORAGE> acc;
  __shared__ __align__(8) RoundOf<MODE> rd;
  const HeavyBricks& hb = bb.heavy;
  for_units(hb, units, bb.status, [&](uint32_t g, uint32_t chunk, bool extra) {
    const int s = batch_scene_of(w, g);
    const BatchScene& S = w.scenes[s];
    brick_unit<MODE, STORAGE>(S.sp, bb.tri_rec + __ldg(bb.tri_prefix + s), S.N, g - __ldg(w.prefix + s), bb.brick_offset + S.brick_base, bb.pair_list,
                              bb.pair_cap, S.ms.l0_surf, nullptr, bb.status, acc, rd, InjGrids{}, nullptr,
                              &hb, g, chunk, extra, FUSE ? bb.mips + s : nullptr,
                              bb.dirty ? bb.dirty + S.brick_base : nullptr);
  });
}

// Persistent grid of a batched kernel: `per_sm` CTAs per SM, but never more
// than fit on an SM at once (a CTA that waits for a slot would start its
// share of the work only after a whole resident CTA has finished).
template <class K>
unsigned resident_grid(K kern, int threads, size_t smem, int sms, int per_sm, uint32_t items) {
  int fit = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, threads, smem) != cudaSuccess || fit < 1) fit = 1;
  const int n = sms * std::min(std::max(per_sm, 1), fit);
  return (unsigned)std::max<uint32_t>(1u, std::min<uint32_t>((uint32_t)n, items));
}

// The same brick work writing RGBA8 level 0 into linear memory (x fastest)
// instead of a surface: the output of vct_voxelize_noalloc.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 7)
    k_bricks_linear(SceneParams sp, int N, const uint32_t* offset, const uint32_t* list,
                    uint32_t cap, uchar4* __restrict__ out, FrameStatus* st, HeavyBricks hb, BrickUnits units) {
  __shared__ Acc acc;
  __shared__ __align__(8) RoundOf<MODE> rd;
  for_units(hb, units, st, [&](uint32_t brick, uint32_t chunk, bool extra) {
    brick_unit<MODE, VCT_STORAGE_RGBA8, false, false>(sp, nullptr, N, brick, offset, list, cap, 0, nullptr, st, acc,
                                                      rd, InjGrids{}, out, &hb, brick, chunk, extra);
  });
}

// CTAs of a kernel resident on one SM.
template <class K>
int resident_per_sm(K kern) {
  int f = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f, kern, kThreads, 0) != cudaSuccess || f < 1) f = 1;
  return f;
}
int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// The filling passes of one renderer's triangles.
cudaError_t fill_lists(const SceneParams& sp, int N, const VoxBuffers& vb, unsigned tri_blocks, cudaStream_t st) {
  cudaError_t e = launch_next(k_bin<true>, tri_blocks, 256, st, sp, N, nullptr, vb.brick_cursor, vb.pair_list,
                              vb.pair_cap, vb.status, vb.big, vb.big_cap, vb.big_count, vb.bin_rec, nullptr);
  if (e != cudaSuccess) return e;
  return launch_next(k_bin_big<true>, dim3(128, kBigSplit), 256, st, N, vb.big, vb.big_cap, vb.big_count, nullptr,
                     vb.brick_cursor, vb.pair_list, vb.pair_cap, nullptr);
}

}  // namespace

cudaError_t launch_voxelize_linear(const SceneParams& sp, int N, int mode, const VoxBuffers& vb, uchar4* out,
                                   cudaStream_t st) {
  const int nb = N / kBrick;
  const size_t n_bricks = (size_t)nb * nb * nb;
  const HeavyBricks& hb = vb.heavy;
  auto* kern = mode == VCT_VOX_CONSERVATIVE ? k_bricks_linear<VCT_VOX_CONSERVATIVE>
                                            : k_bricks_linear<VCT_VOX_REF_RASTER2X>;
  const unsigned grid = (unsigned)std::min<size_t>((size_t)sm_count() * resident_per_sm(kern), n_bricks + hb.item_cap);
  cudaError_t e = cudaMemsetAsync(vb.brick_count, 0, n_bricks * sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(vb.big_count, 0, sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
  const unsigned tri_blocks = (sp.total_tris + 255) / 256;
  const dim3 big_grid(128, kBigSplit);
  if (tri_blocks) {
    k_bin<false><<<tri_blocks, 256, 0, st>>>(sp, N, vb.brick_count, nullptr, nullptr, 0, vb.status, vb.big, vb.big_cap,
                                             vb.big_count, vb.bin_rec, nullptr);
    e = launch_next(k_bin_big<false>, big_grid, 256, st, N, vb.big, vb.big_cap, vb.big_count, vb.brick_count, nullptr,
                    nullptr, 0u, nullptr);
    if (e != cudaSuccess) return e;
  }
  ScanFuse fuse;
  std::memset(&fuse, 0, sizeof(fuse));
  fuse.hb = hb;
  fuse.units = brick_units(vb.units, (uint32_t)n_bricks, nullptr, nullptr);
  fuse.cap = vb.pair_cap;
  fuse.slots = grid;
  fuse.total_copy = &vb.status->pair_total;
  e = launch_exclusive_scan(vb.brick_count, vb.brick_offset, vb.brick_cursor, n_bricks, vb.scan_tmp, st, nullptr,
                            &fuse);
  if (e != cudaSuccess) return e;
  if (tri_blocks) {
    e = fill_lists(sp, N, vb, tri_blocks, st);
    if (e != cudaSuccess) return e;
  }
  return launch_next(kern, grid, kThreads, st, sp, N, vb.brick_offset, vb.pair_list, vb.pair_cap, out, vb.status, hb,
                     fuse.units);
}

// Calls f(mode tag, storage tag) for the brick kernel a frame uses.
template <class F>
void dispatch_bricks(int mode, int storage, bool attr, F&& f) {
  using RAS = std::integral_constant<int, VCT_VOX_REF_RASTER2X>;
  using SAT = std::integral_constant<int, VCT_VOX_CONSERVATIVE>;
  using R8 = std::integral_constant<int, VCT_STORAGE_RGBA8>;
  using F16 = std::integral_constant<int, VCT_STORAGE_RGBA16F>;
  using ATR = std::integral_constant<int, kStorageAttr>;
  if (mode == VCT_VOX_CONSERVATIVE) {
    if (attr) f(SAT(), ATR());
    else if (storage == VCT_STORAGE_RGBA8) f(SAT(), R8());
    else f(SAT(), F16());
  } else {
    if (attr) f(RAS(), ATR());
    else if (storage == VCT_STORAGE_RGBA8) f(RAS(), R8());
    else f(RAS(), F16());
  }
}

cudaError_t launch_voxelize(const SceneParams& sp, int N, int mode, int storage, const VoxBuffers& vb,
                            cudaSurfaceObject_t l0, cudaStream_t st, int* launches, const InjGrids* inj) {
  int nl = 0;
  const int nb = N / kBrick;
  const size_t n_bricks = (size_t)nb * nb * nb;
  const int sms = sm_count();
  const bool fuse_mips = vb.mips && !inj && (storage == VCT_STORAGE_RGBA8 || storage == VCT_STORAGE_RGBA16F);
  int fit = 1;
  dispatch_bricks(mode, storage, inj != nullptr, [&](auto mode_tag, auto storage_tag) {
    constexpr int M = decltype(mode_tag)::value, S = decltype(storage_tag)::value;
    static const int plain = resident_per_sm(k_bricks<M, S>);
    fit = plain;
    if constexpr (S == VCT_STORAGE_RGBA8 || S == VCT_STORAGE_RGBA16F) {
      static const int fused = resident_per_sm(k_bricks<M, S, true>);
      if (fuse_mips) fit = fused;
    }
  });
  const uint8_t* dirty = inj || vb.counts ? nullptr : vb.dirty;
  const BrickUnits units = brick_units(vb.units, (uint32_t)n_bricks, dirty, vb.big_count);
  cudaError_t e = cudaSuccess;
  const unsigned tri_blocks = (sp.total_tris + 255) / 256;
  if (tri_blocks) {
    k_bin<false><<<tri_blocks, 256, 0, st>>>(sp, N, vb.brick_count, nullptr, nullptr, 0, vb.status, vb.big,
                                             vb.big_cap, vb.big_count, vb.bin_rec, vb.tri_rec);
    e = launch_next(k_bin_big<false>, dim3(128, kBigSplit), 256, st, N, vb.big, vb.big_cap, vb.big_count,
                    vb.brick_count, nullptr, nullptr, 0u, nullptr);
    if (e != cudaSuccess) return e;
    nl += 2;
  }
  // Offsets, pair_total <- offset[n_bricks], and the dense-brick plan
  // against the brick CTAs resident at once.
  const HeavyBricks& hb = vb.heavy;
  ScanFuse fuse;
  std::memset(&fuse, 0, sizeof(fuse));
  fuse.hb = hb;
  fuse.units = units;
  fuse.cap = vb.pair_cap;
  fuse.slots = (uint32_t)(sms * fit);
  fuse.total_copy = &vb.status->pair_total;
  fuse.big_total = &vb.status->bigtri_total;
  fuse.big_count = vb.big_count;
  fuse.clear = true;
  e = launch_exclusive_scan(vb.brick_count, vb.brick_offset, vb.brick_cursor, n_bricks, vb.scan_tmp, st, &nl, &fuse);
  if (e != cudaSuccess) return e;
  if (tri_blocks) {
    e = fill_lists(sp, N, vb, tri_blocks, st);
    if (e != cudaSuccess) return e;
    nl += 2;
  }
  const InjGrids g = inj ? *inj : InjGrids{};
  void* lin = inj ? nullptr : vb.level0_lin;
  BrickMips bm;
  std::memset(&bm, 0, sizeof(bm));
  if (fuse_mips) bm = *vb.mips;
  bm.dirty = inj ? nullptr : vb.dirty;  // (kernel parameter of every brick kernel)
  const unsigned grid = (unsigned)std::min<size_t>((size_t)sms * fit, n_bricks + (hb.slot ? hb.item_cap : 0u));
  dispatch_bricks(mode, storage, inj != nullptr, [&](auto mode_tag, auto storage_tag) {
    constexpr int M = decltype(mode_tag)::value, S = decltype(storage_tag)::value;
    if constexpr (S == VCT_STORAGE_RGBA8 || S == VCT_STORAGE_RGBA16F) {
      if (fuse_mips) {
        e = launch_next(k_bricks<M, S, true>, grid, kThreads, st, sp, N, vb.brick_offset, vb.pair_list, vb.pair_cap, l0, vb.counts, vb.status, g, lin, hb, units, vb.tri_rec, bm);
        return;
      }
    }
    e = launch_next(k_bricks<M, S>, grid, kThreads, st, sp, N, vb.brick_offset, vb.pair_list, vb.pair_cap, l0, vb.counts, vb.status, g, lin, hb, units, vb.tri_rec, bm);
  });
  if (e != cudaSuccess) return e;
  ++nl;
  if (launches) *launches += nl;
  return cudaGetLastError();
}

size_t heavy_slot_bytes(int storage) {
  return storage == kStorageAttr          ? sizeof(AccT<kStorageAttr>)
         : storage == VCT_STORAGE_RGBA16F ? sizeof(AccT<VCT_STORAGE_RGBA16F>)
                                          : sizeof(AccT<VCT_STORAGE_RGBA8>);
}

}  // namespace vct

namespace vct {

// Batched voxelizer: the same passes as launch_voxelize, each one launch
// over every scene of the batch (brick arrays concatenated, one scan).
cudaError_t launch_voxelize_batch(const BatchWork& tris, const BatchWork& bricks, uint32_t total_bricks, int mode,
                                  int storage, const BatchBuffers& bb, uint32_t* scan_tmp, const BatchShape& shape,
                                  int sms, cudaStream_t st, int* launches) {
  int nl = 0;
  const HeavyBricks& hb = bb.heavy;
  // The persistent brick grid (bricks + at most item_cap extra chunks).
  unsigned grid = 1;
  const bool fuse_mips = bb.mips != nullptr && storage == VCT_STORAGE_RGBA8;
  dispatch_bricks(mode, storage, false, [&](auto mode_tag, auto storage_tag) {
    constexpr int M = decltype(mode_tag)::value, S = decltype(storage_tag)::value;
    grid = fuse_mips ? resident_grid(k_bricks_batch<M, S, true>, kThreads, 0, sms, shape.bricks_ctas_per_sm,
                                bricks.total + (hb.slot ? hb.item_cap : 0u))
                : resident_grid(k_bricks_batch<M, S>, kThreads, 0, sms, shape.bricks_ctas_per_sm,
                                bricks.total + (hb.slot ? hb.item_cap : 0u));
  });
  cudaError_t e = cudaSuccess;
  const unsigned bin_grid = resident_grid(k_bin_batch<false>, 256, 0, sms, shape.bin_ctas_per_sm,
                                          (tris.total + 255) / 256);
  const dim3 big_grid(128, kBigSplit);
  if (tris.total) {
    k_bin_batch<false><<<bin_grid, 256, 0, st>>>(tris, bb);
    e = launch_next(k_bin_big<false>, big_grid, 256, st, 0, bb.big, bb.big_cap, bb.big_count, bb.brick_count, nullptr,
                    nullptr, 0u, tris.scenes);
    if (e != cudaSuccess) return e;
    nl += 2;
  }
  // Offsets, pair_total, the dense-brick plan against the persistent grid's
  // CTAs, and the bricks with work.
  const BrickUnits units = brick_units(bb.units, total_bricks, bb.dirty, bb.big_count);
  ScanFuse fuse;
  std::memset(&fuse, 0, sizeof(fuse));
  fuse.hb = hb;
  fuse.units = units;
  fuse.cap = bb.pair_cap;
  fuse.slots = grid;
  fuse.total_copy = &bb.status->pair_total;
  fuse.big_total = &bb.status->bigtri_total;
  fuse.big_count = bb.big_count;
  fuse.clear = true;
  e = launch_exclusive_scan(bb.brick_count, bb.brick_offset, bb.brick_cursor, total_bricks, scan_tmp, st, &nl, &fuse);
  if (e != cudaSuccess) return e;
  if (tris.total) {
    e = launch_next(k_bin_batch<true>, bin_grid, 256, st, tris, bb);
    if (e != cudaSuccess) return e;
    e = launch_next(k_bin_big<true>, big_grid, 256, st, 0, bb.big, bb.big_cap, bb.big_count, nullptr, bb.brick_cursor,
                    bb.pair_list, bb.pair_cap, tris.scenes);
    if (e != cudaSuccess) return e;
    nl += 2;
  }
  dispatch_bricks(mode, storage, false, [&](auto mode_tag, auto storage_tag) {
    constexpr int M = decltype(mode_tag)::value, S = decltype(storage_tag)::value;
    e = launch_next(fuse_mips ? k_bricks_batch<M, S, true> : k_bricks_batch<M, S>, grid, kThreads, st, bricks, bb, units);
  });
  if (e != cudaSuccess) return e;
  ++nl;
  if (launches) *launches += nl;
  return cudaGetLastError();
}

}  // namespace vct

namespace vct {
namespace {

// Deferred light injection (no reference counterpart: the reference shades
// every fragment while voxelizing, voxelize.frag:124-153).  Each occupied
// voxel is lit at its centre (grid space (2x+1)/N - 1) with its mean normal
// and the same per-light terms as voxelize.frag:128-143:
//   colour = clamp(albedo * sum_i color_i * intensity_i * max(n.l_i, 0) /
//                  (1 + d_i^2) + emission, 0, 1),  alpha = mean alpha,
// stored as RGBA8 rounded to nearest.
//
// Bound by memory: 12 bytes a voxel (emission read, level 0 written to its
// surface and its linear copy), most voxels being empty.  A thread takes four
// voxels of a row, 16 bytes of each grid at a time.  The room's walls leave an
// occupied voxel to nearly every warp, so the groups that hold one are queued
// and lit a full warp at a time, by resident CTAs whose queues seldom run
// short.  256^3, 300,000 occupied: 153 us with a thread a voxel, 76 by fours,
// 72 at 48 warps an SM, 48 with the queue (40 warps, no spills; 48 spill: 68).
__device__ __forceinline__ uint32_t inject_voxel(const SceneParams& sp, float inv, int x, int y, int z, uint32_t ep,
                                                 uint32_t ap, uint32_t np) {
  const float k = 1.0f / 255.0f;
  const uchar4 e = make_uchar4(ep & 255u, ep >> 8 & 255u, ep >> 16 & 255u, ep >> 24);
  const uchar4 a = make_uchar4(ap & 255u, ap >> 8 & 255u, ap >> 16 & 255u, ap >> 24);
  const uchar4 nq = make_uchar4(np & 255u, np >> 8 & 255u, np >> 16 & 255u, np >> 24);
  const V3 nn = normalize(v3(nq.x * k * 2.0f - 1.0f, nq.y * k * 2.0f - 1.0f, nq.z * k * 2.0f - 1.0f));
  const V3 pos = v3(((float)x + 0.5f) * inv - 1.0f, ((float)y + 0.5f) * inv - 1.0f, ((float)z + 0.5f) * inv - 1.0f);
  V3 lit = v3(0.f, 0.f, 0.f);
  const int nl = min(sp.n_lights, kMaxLights);
  for (int l = 0; l < nl; ++l) {
    const vct_point_light& L = sp.lights[l];
    const V3 lp = v3(L.position[0] / sp.cube_size, L.position[1] / sp.cube_size, L.position[2] / sp.cube_size);
    const V3 dl = lp - pos;
    const float d = length(dl);
    const float cs = fmaxf(dot(nn, normalize(dl)), 0.0f);
    lit = lit + v3(L.color[0], L.color[1], L.color[2]) * (cs * (1.0f / (1.0f + d * d)) * L.intensity);
  }
  const V3 c = mulv(v3(a.x * k, a.y * k, a.z * k), lit) + v3(e.x * k, e.y * k, e.z * k);
  auto q = [](float v) { return __float2uint_rz(clamp01(v) * 255.0f + 0.5f); };
  return q(c.x) | q(c.y) << 8 | q(c.z) << 16 | (uint32_t)a.w << 24;
}

// (N: a power of two, at least 8.)
__global__ void __launch_bounds__(256, 5) k_inject(SceneParams sp, int N, InjGrids g, cudaSurfaceObject_t l0,
                                                uint4* __restrict__ l0_lin) {
  __shared__ uint32_t s_queue[8][64];
  uint32_t* queue = s_queue[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, sh = __ffs(N) - 1;
  const uint32_t total = 1u << (3 * sh - 2);  // (a multiple of 32: whole warps)
  const float inv = 2.0f / (float)N;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  int queued = 0;
  for (;;) {
    while (queued < 32 && i < total) {
      const int x = (int)(4u * i) & (N - 1), y = (int)(i >> (sh - 2)) & (N - 1), z = (int)(i >> (2 * sh - 2));
      uint4 e;
      surf3Dread(&e, g.emission, x * 4, y, z);
      const bool any = (e.x | e.y | e.z | e.w) >> 24 != 0u;  // (occupied: its emission's alpha)
      if (!any) {
        surf3Dwrite(make_uint4(0u, 0u, 0u, 0u), l0, x * 4, y, z);
        if (l0_lin) l0_lin[i] = make_uint4(0u, 0u, 0u, 0u);
      }
      const unsigned some = __ballot_sync(0xffffffffu, any);
      if (any) queue[queued + __popc(some & ((1u << lane) - 1u))] = i;
      queued += __popc(some);
      i += gridDim.x * blockDim.x;
    }
    const int m = min(queued, 32);
    if (m == 0) return;
    __syncwarp();
    queued -= m;
    if (lane < m) {
      const uint32_t v = queue[queued + lane];
      const int x = (int)(4u * v) & (N - 1), y = (int)(v >> (sh - 2)) & (N - 1), z = (int)(v >> (2 * sh - 2));
      uint4 e, a, n, o = make_uint4(0u, 0u, 0u, 0u);
      surf3Dread(&e, g.emission, x * 4, y, z);
      surf3Dread(&a, g.albedo, x * 4, y, z);
      surf3Dread(&n, g.normal, x * 4, y, z);
#pragma unroll 1
      for (int j = 0; j < 4; ++j) {
        uint32_t c = 0u;
        if (e.x >> 24) c = inject_voxel(sp, inv, x + j, y, z, e.x, a.x, n.x);
        o = make_uint4(o.y, o.z, o.w, c);
        e = make_uint4(e.y, e.z, e.w, 0u);
        a = make_uint4(a.y, a.z, a.w, 0u);
        n = make_uint4(n.y, n.z, n.w, 0u);
      }
      surf3Dwrite(o, l0, x * 4, y, z);
      if (l0_lin) l0_lin[v] = o;
    }
    __syncwarp();  // the entries are read before their place is written again
  }
}

}  // namespace

cudaError_t launch_inject(const SceneParams& sp, int N, const InjGrids& g, cudaSurfaceObject_t l0, uchar4* l0_lin,
                          cudaStream_t st, int* launches) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t total = (size_t)N * N * N / 4;
  const unsigned grid = (unsigned)std::min<size_t>((total + 255) / 256, (size_t)sms * 5);
  k_inject<<<grid, 256, 0, st>>>(sp, N, g, l0, reinterpret_cast<uint4*>(l0_lin));
  if (launches) ++*launches;
  return cudaGetLastError();
}

}  // namespace vct
