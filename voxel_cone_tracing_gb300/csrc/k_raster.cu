// k_raster.cu -- G-buffer production: the forward raster of
// Renderer::visualize (renderer.cpp:355-390) with voxel_cone_tracing.vert
// :22-27, as CUDA kernels.
//
// The reference shades every fragment that passes GL_LESS at its time; the
// final image is the nearest surface (first drawn on equal depth).  Here the
// visible surface is found first and shaded once:
//   k_gb_setup  -- per triangle: world = M*p, clip = (P*V)*world (FP32, fixed
//                  order); triangles crossing the near plane or a guard band
//                  of |x|,|y| <= 16w are clipped (Sutherland-Hodgman) and
//                  fanned; vertices snapped to 1/256 pixel; triangles whose
//                  pixel box holds <= 64 pixels are rasterised right here,
//                  larger ones become records.
//   k_gb_big    -- a warp per 32x32-pixel tile of a record's box.
//   coverage    -- integer edge functions at pixel centres, top-left rule;
//                  depth = FP32 z_window interpolated in screen space; the
//                  visibility buffer keeps min((depth bits << 32) | triangle
//                  id) via 64-bit atomicMin (ties -> earlier triangle).
//   k_gb_resolve -- per pixel: perspective-correct barycentrics of the
//                  visible triangle -> world position, interpolated world
//                  normal (not renormalised), material id.
#include <algorithm>
#include <type_traits>

#include "vct_internal.h"
#include "vct_math.cuh"
#include "vct_snap.h"
#include "vct_tiles.h"

namespace vct {
namespace {

// The box a setup thread rasters itself: its loop is serial, a record costs an
// atomic and a warp of k_gb_big.  G-buffer of 500,000 triangles at 1920x1080 and
// 120,000 at 1367x771: 8 pixels 172 and 174 us, 16 129 and 96, 32 110 and 89,
// 64 106 and 84.
constexpr int kSmallPixels = 64;
constexpr int kAcross = 2;    // blocks of a row in flight
constexpr int kSetup = 128;   // threads of a setup block
constexpr float kGuard = 16.0f;

// A screen triangle: counter-clockwise, snapped vertices, window depths.
struct BigRec {
  int X[3], Y[3];
  float z[3];
  float farea;
  uint32_t tri;
  int tl;              // bit k: edge k keeps the samples on it
  int x0, y0, x1, y1;  // pixel bbox (inclusive)
  uint32_t tw;         // tiles across
  uint32_t scene;      // scene of a batch (0 for one renderer)
};

__device__ __forceinline__ int find_instance(const SceneParams& sp, uint32_t t) {
  int lo = 0, hi = (int)sp.n_instances - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (sp.inst[mid].tri_base <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

struct CV { float c[4]; };

__device__ __forceinline__ void vertex_clip(const DevInstance& in, const float* PV, uint32_t vi, float w[3], CV& cv,
                                            float4* a_out = nullptr, float4* b_out = nullptr) {
  const float4* vp = reinterpret_cast<const float4*>(in.verts + vi);
  const float4 a = __ldg(vp), b = __ldg(vp + 1);
  for (int r = 0; r < 3; ++r) w[r] = xform_row(in.M, r, a.x, a.y, a.z);
  for (int r = 0; r < 4; ++r) {
    float t = rmul(PV[0 * 4 + r], w[0]);
    t = radd(t, rmul(PV[1 * 4 + r], w[1]));
    t = radd(t, rmul(PV[2 * 4 + r], w[2]));
    cv.c[r] = radd(t, PV[3 * 4 + r]);
  }
  if (a_out) *a_out = a;
  if (b_out) *b_out = b;
}

__device__ __forceinline__ float plane_eval(int pl, const CV& v) {
  switch (pl) {
    case 0: return radd(v.c[2], v.c[3]);
    case 1: return rsub(rmul(kGuard, v.c[3]), v.c[0]);
    case 2: return radd(rmul(kGuard, v.c[3]), v.c[0]);
    case 3: return rsub(rmul(kGuard, v.c[3]), v.c[1]);
    default: return radd(rmul(kGuard, v.c[3]), v.c[1]);
  }
}

// The visibility key of depth zz: ~0 (never stored) past the far plane.
__device__ __forceinline__ unsigned long long depth_key(float zz, uint32_t tri) {
  if (!(zz < 1.0f)) return ~0ull;
  if (!(zz > 0.0f)) zz = 0.0f;
  return ((unsigned long long)__float_as_uint(zz) << 32) | tri;
}

// The edge functions of a triangle at a pixel centre, each lowered by one
// where the edge does not keep the samples on it: inside = none negative.
template <class T>
struct Edges {
  T w[3];
  T dx[3], dy[3];  // per pixel across, per pixel up
  int on[3];       // what w was lowered by
  __device__ __forceinline__ void at(const BigRec& r, int px, int py) {
    const T sx = (T)(256 * px + 128), sy = (T)(256 * py + 128);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int a = (k + 1) % 3, b = (k + 2) % 3;  // edge k: vertex k + 1 -> vertex k + 2
      const T ex = (T)r.X[b] - r.X[a], ey = (T)r.Y[b] - r.Y[a];
      on[k] = (r.tl >> k) & 1 ? 0 : 1;
      w[k] = ex * (sy - r.Y[a]) - ey * (sx - r.X[a]) - on[k];
      dx[k] = -ey * 256;
      dy[k] = ex * 256;
    }
  }
  __device__ __forceinline__ bool inside() const { return (w[0] | w[1] | w[2]) >= 0; }
};
__device__ __forceinline__ float to_float(int v) { return __int2float_rn(v); }
__device__ __forceinline__ float to_float(long long v) { return __ll2float_rn(v); }

template <class T>
__device__ __forceinline__ unsigned long long pixel_key(const BigRec& r, const Edges<T>& e) {
  const float b1 = rdiv(to_float(e.w[1] + e.on[1]), r.farea), b2 = rdiv(to_float(e.w[2] + e.on[2]), r.farea);
  float zz = radd(r.z[0], rmul(b1, rsub(r.z[1], r.z[0])));
  zz = radd(zz, rmul(b2, rsub(r.z[2], r.z[0])));
  return depth_key(zz, r.tri);
}

// Rasterises the record's whole box, one thread.
template <class T>
__device__ __forceinline__ void raster_box(const BigRec& r, unsigned long long* vis, int W) {
  Edges<T> e;
  e.at(r, r.x0, r.y0);
  for (int py = r.y0; py <= r.y1; ++py) {
    Edges<T> q = e;
    for (int px = r.x0; px <= r.x1; ++px) {
      if (q.inside()) {
        const unsigned long long key = pixel_key(r, q);
        if (key != ~0ull) atomicMin(vis + (size_t)py * W + px, key);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) q.w[k] += q.dx[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) e.w[k] += e.dy[k];
  }
}

// Screen coordinates while a triangle is set up: 32 bits hold those of a frame
// within kSnapPixels each way (|n| <= 64: below 2^28, their differences too).
template <bool WIDE>
using Coord = typename std::conditional<WIDE, long long, int>::type;

// 1/256-pixel coordinate of normalised device coordinate n on `pixels` pixels.
template <bool WIDE>
__device__ __forceinline__ Coord<WIDE> snap_ndc(float n, int pixels) {
  if constexpr (WIDE) {
    return __double2ll_rn(__dmul_rn(__dadd_rn((double)n, 1.0), (double)pixels * 128.0));
  } else {
    const int K = pixels * 128;
    bool close;
    const int v = snap_scaled(n, (uint32_t)K, close);
    if (!close) return v;
    return (int)__double2ll_rn(__dmul_rn(__dadd_rn((double)n, 1.0), (double)K));
  }
}

// Set up one (possibly clipped) screen triangle; raster it here if small.
template <bool WIDE>
__device__ __forceinline__ void raster_subtri(const CV v[3], int W, int H, uint32_t tri, const RasterBuffers& rb,
                                              uint32_t scene) {
  typedef Coord<WIDE> C;
  BigRec r;
  C X[3], Y[3];
  for (int k = 0; k < 3; ++k) {
    if (!(v[k].c[3] > 0.0f)) return;
    const float nx = rdiv(v[k].c[0], v[k].c[3]), ny = rdiv(v[k].c[1], v[k].c[3]), nz = rdiv(v[k].c[2], v[k].c[3]);
    if (!(fabsf(nx) <= 64.0f) || !(fabsf(ny) <= 64.0f) || !(nz == nz)) return;
    X[k] = snap_ndc<WIDE>(nx, W);
    Y[k] = snap_ndc<WIDE>(ny, H);
    r.z[k] = radd(rmul(0.5f, nz), 0.5f);
  }
  const long long ax = X[1] - X[0], ay = Y[1] - Y[0], bx = X[2] - X[0], by = Y[2] - Y[0];
  long long area = ax * by - ay * bx;
  if (area == 0) return;
  if (area < 0) {
    C t = X[1]; X[1] = X[2]; X[2] = t;
    t = Y[1]; Y[1] = Y[2]; Y[2] = t;
    float tz = r.z[1]; r.z[1] = r.z[2]; r.z[2] = tz;
    area = -area;
  }
  // the pixels whose centres (256 p + 128) lie in the box
  const C minx = min(X[0], min(X[1], X[2])), maxx = max(X[0], max(X[1], X[2]));
  const C miny = min(Y[0], min(Y[1], Y[2])), maxy = max(Y[0], max(Y[1], Y[2]));
  r.x0 = (int)max((C)0, (minx + 127) >> 8);
  r.x1 = (int)min((C)(W - 1), (maxx - 128) >> 8);
  r.y0 = (int)max((C)0, (miny + 127) >> 8);
  r.y1 = (int)min((C)(H - 1), (maxy - 128) >> 8);
  if (r.x1 < r.x0 || r.y1 < r.y0) return;
  for (int k = 0; k < 3; ++k) {
    r.X[k] = (int)X[k];
    r.Y[k] = (int)Y[k];
  }
  r.farea = __ll2float_rn(area);
  r.tl = (top_left(X[1], Y[1], X[2], Y[2]) ? 1 : 0) | (top_left(X[2], Y[2], X[0], Y[0]) ? 2 : 0) |
         (top_left(X[0], Y[0], X[1], Y[1]) ? 4 : 0);
  r.tri = tri;
  const int nx = r.x1 - r.x0 + 1, ny = r.y1 - r.y0 + 1;
  if (nx * ny <= kSmallPixels) {
    // (within 2^14 the products of two differences stay below 2^29)
    if (!WIDE && maxx - minx <= (1 << 14) && maxy - miny <= (1 << 14)) raster_box<int>(r, rb.vis, W);
    else raster_box<long long>(r, rb.vis, W);
    return;
  }
  r.scene = scene;
  // Records and tiles are counted in one word, so the first tiles ascend with
  // the records and need no scan.  The lanes with a single tile, most of them,
  // share one atomic.
  r.tw = tiles_across(r.x0, r.x1);
  const uint32_t tiles = tiles_of(r.x0, r.y0, r.x1, r.y1);
  unsigned long long at;
  if (tiles == 1) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, lead = __ffs((int)m) - 1;
    unsigned long long base = 0;
    if (lane == lead) base = atomicAdd(rb.big_count, big_count_of(1, 1) * (unsigned)__popc(m));
    at = __shfl_sync(m, base, lead) + big_count_of(1, 1) * (unsigned)__popc(m & ((1u << lane) - 1u));
  } else {
    at = atomicAdd(rb.big_count, big_count_of(1, tiles));
  }
  const uint32_t slot = big_records(at);
  if (slot >= rb.big_cap) return;  // (reported; the frame is encoded again)
  reinterpret_cast<BigRec*>(rb.big)[slot] = r;
  rb.big_first[slot] = big_tiles(at);
}

// The clipped triangle's fan, called, not inlined: its polygons live in local
// memory, and few triangles need it.
template <bool WIDE>
__device__ __noinline__ void raster_clipped(const CV cv[3], int W, int H, uint32_t t, const RasterBuffers& rb,
                                            uint32_t scene) {
  CV a[10], b[10];
  int n = 3;
  for (int k = 0; k < 3; ++k) a[k] = cv[k];
#pragma unroll 1
  for (int pl = 0; pl < 5; ++pl) {
    int m = 0;
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const CV p0 = a[i], p1 = a[(i + 1) % n];
      const float d0 = plane_eval(pl, p0), d1 = plane_eval(pl, p1);
      const bool in0 = d0 >= 0.0f, in1 = d1 >= 0.0f;
      if (in0) b[m++] = p0;
      if (in0 != in1) {
        const float tt = rdiv(d0, rsub(d0, d1));
        CV q;
        for (int c = 0; c < 4; ++c) q.c[c] = radd(p0.c[c], rmul(tt, rsub(p1.c[c], p0.c[c])));
        b[m++] = q;
      }
    }
    n = m;
    for (int i = 0; i < n; ++i) a[i] = b[i];
    if (n < 3) return;
  }
#pragma unroll 1
  for (int k = 1; k + 1 < n; ++k) {
    const CV tri3[3] = {a[0], a[k], a[k + 1]};
    raster_subtri<WIDE>(tri3, W, H, t, rb, scene);
  }
}

template <bool WIDE>
__device__ __forceinline__ void setup_tri(const SceneParams& sp, const CameraParams& cp, const RasterBuffers& rb,
                                          uint32_t t, uint32_t scene) {
  if (t >= sp.total_tris) return;
  const DevInstance& in = sp.inst[find_instance(sp, t)];
  const uint32_t lt = t - in.tri_base;
  CV cv[3];
  float w[3];
  for (int k = 0; k < 3; ++k) vertex_clip(in, cp.PV, __ldg(in.indices + 3 * (size_t)lt + k), w, cv[k]);
  bool all_in = true;
  for (int pl = 0; pl < 5; ++pl)
    for (int k = 0; k < 3; ++k)
      if (!(plane_eval(pl, cv[k]) >= 0.0f)) all_in = false;
  if (all_in) raster_subtri<WIDE>(cv, cp.W, cp.H, t, rb, scene);
  else raster_clipped<WIDE>(cv, cp.W, cp.H, t, rb, scene);
}

// Latency of the instance, index and vertex loads, so registers decide (64: 32
// warps an SM): vertices are snapped without FP64, a rate-limited unit here;
// small boxes take 32-bit stepped edge functions and fire-and-forget atomics
// (reading the visibility word first, to skip the atomic, stalled on every
// pixel); the clipper is a call.  500,000 triangles, 1920x1080: 86 us with
// FP64 and the clipper inline (98 registers), 38 now.  WIDE (snap_wide): with
// FP64 and 64-bit coordinates.
template <bool WIDE>
__global__ void __launch_bounds__(kSetup, 8) k_gb_setup(SceneParams sp, CameraParams cp, RasterBuffers rb) {
  setup_tri<WIDE>(sp, cp, rb, blockIdx.x * blockDim.x + threadIdx.x, 0u);
}

// The pixel slice of one batch scene in the batch-wide raster buffers.
__device__ __forceinline__ RasterBuffers scene_rb(const RasterBuffers& rb, const BatchScene& S) {
  RasterBuffers r = rb;
  r.vis = rb.vis + S.px_base;
  r.gb_pos = rb.gb_pos + S.px_base;
  r.gb_nrm = rb.gb_nrm + S.px_base;
  return r;
}

// (a batch's frames are within kSnapPixels)
__global__ void __launch_bounds__(kSetup, 8) k_gb_setup_batch(BatchWork w, RasterBuffers rb) {
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < w.total; g += gridDim.x * blockDim.x) {
    const int s = batch_scene_of(w, g);
    const BatchScene& S = w.scenes[s];
    setup_tri<false>(S.sp, w.cams[s], scene_rb(rb, S), g - __ldg(w.prefix + s), (uint32_t)s);
  }
}

// The last of n ascending values that is not above x (the first one is not),
// found by a warp.
__device__ __forceinline__ uint32_t warp_last_not_above(const unsigned long long* v, uint32_t n,
                                                        unsigned long long x) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t step = (hi - lo + 31) / 32, i = lo + lane * step;
    const unsigned below = __ballot_sync(0xffffffffu, i < hi && v[i] <= x);
    lo += (31 - __clz((int)below)) * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

// The large triangles' tiles, a warp each, 8x4 pixels at a time with the edge
// functions stepped from block to block.  A warp finds its tile's record in
// the ascending first tiles by a 32-way search (three or four probes); a tile
// wholly outside an edge stops there.  Bound by the chain of loads to the
// record and by the atomics' issue, which is why they return nothing.  16x16
// tiles with a thread to a pixel, a scan kernel for their offsets and a binary
// search in every thread took 75 + 5 us (1920x1080, 500,000 triangles), this
// takes 20; 16 scenes in a batch 752 + 102 -> 95.  Lists of tiles written by
// the setup thread were no alternative: one thread writes a whole screen's
// (64x64 tiles 155 us for all of the G-buffer, 32x32 210).
__global__ void __launch_bounds__(256) k_gb_big(RasterBuffers rb, int W, const BatchScene* scenes) {
  follows_previous();
  const uint32_t records = big_records(*rb.big_count), listed = min(records, rb.big_cap);
  unsigned long long total = big_tiles(*rb.big_count);
  const int lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    rb.status->big_total = records;
    rb.status->big_tiles = (uint32_t)min(total, 0xffffffffull);
  }
  if (!listed) return;
  if (listed < records) {  // a full list (reported by big_total): its records' tiles
    const BigRec& last = reinterpret_cast<const BigRec*>(rb.big)[listed - 1];
    total = rb.big_first[listed - 1] + tiles_of(last.x0, last.y0, last.x1, last.y1);
  }
  // few tiles: up to 8 warps on one, each taking every so many-th row of blocks
  const uint32_t warps = gridDim.x * 8;
  int sh = 0;
  while (sh < 3 && total <= warps >> (sh + 1)) ++sh;
  for (unsigned long long j = blockIdx.x * 8 + (threadIdx.x >> 5); j >> sh < total; j += warps) {
    const unsigned long long t = j >> sh;
    const int strip = (int)((unsigned)j & ((1u << sh) - 1)) * 4, step = 4 << sh;
    const uint32_t n = warp_last_not_above(rb.big_first, listed, t);
    const BigRec r = reinterpret_cast<const BigRec*>(rb.big)[n];
    int x0, y0;
    if (!tile_origin(t - rb.big_first[n], r.tw, r.x0, r.y0, r.y1, x0, y0)) continue;
    unsigned long long* vis = rb.vis;
    int w = W;
    if (scenes) {  // a batch: the record's scene
      vis += scenes[r.scene].px_base;
      w = scenes[r.scene].W;
    }
    const int x1 = min(r.x1, x0 + kTile - 1), y1 = min(r.y1, y0 + kTile - 1);
    Edges<long long> e;
    e.at(r, x0, y0);
    bool out = false;  // an edge with the whole tile outside
#pragma unroll
    for (int k = 0; k < 3; ++k)
      out |= e.w[k] + max(e.dx[k] * (x1 - x0), 0ll) + max(e.dy[k] * (y1 - y0), 0ll) < 0;
    if (out) continue;
    const int lx = lane & 7, ly = lane >> 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      e.w[k] += e.dx[k] * lx + e.dy[k] * (ly + strip);
      e.dx[k] *= 8;
      e.dy[k] *= step;
    }
#pragma unroll 1
    for (int py = y0 + strip + ly; py - ly <= y1; py += step) {
      Edges<long long> q = e;
#pragma unroll 1
      for (int px = x0 + lx; px - lx <= x1; px += 8 * kAcross) {
        unsigned long long key[kAcross], *slot = vis + (size_t)py * w + px;
#pragma unroll
        for (int u = 0; u < kAcross; ++u) {
          key[u] = ~0ull;
          if (q.inside() && px + 8 * u <= x1 && py <= y1) key[u] = pixel_key(r, q);
#pragma unroll
          for (int k = 0; k < 3; ++k) q.w[k] += q.dx[k];
        }
#pragma unroll
        for (int u = 0; u < kAcross; ++u)
          if (key[u] != ~0ull) atomicMin(slot + 8 * u, key[u]);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) e.w[k] += e.dy[k];
    }
  }
}

__device__ __forceinline__ void resolve_px(const SceneParams& sp, const CameraParams& cp, const RasterBuffers& rb,
                                           int px, int py) {
  if (px >= cp.W || py >= cp.H) return;
  const size_t p = (size_t)py * cp.W + px;
  const unsigned long long key = rb.vis[p];
  if (key == ~0ull) {
    rb.gb_pos[p] = make_float4(0.f, 0.f, 0.f, __uint_as_float(0xffffffffu));
    rb.gb_nrm[p] = make_float4(0.f, 0.f, 0.f, __uint_as_float(0xffffffffu));
    return;
  }
  const uint32_t t = (uint32_t)(key & 0xffffffffull);
  const DevInstance& in = sp.inst[find_instance(sp, t)];
  const uint32_t lt = t - in.tri_base;
  CV cv[3];
  V3 wp[3], nn[3];
  for (int k = 0; k < 3; ++k) {
    float w[3];
    float4 a, b;
    vertex_clip(in, cp.PV, __ldg(in.indices + 3 * (size_t)lt + k), w, cv[k], &a, &b);
    wp[k] = v3(w[0], w[1], w[2]);
    nn[k] = normalize(nm_mul(in.NM, a.w, b.x, b.y));
  }
  // Perspective-correct barycentrics: sum b_k (x_k - px w_k) = 0, sum b_k
  // (y_k - py w_k) = 0, sum b_k = 1 (GL smooth interpolation).
  const float pxn = ((float)px + 0.5f) * 2.0f / (float)cp.W - 1.0f;
  const float pyn = ((float)py + 0.5f) * 2.0f / (float)cp.H - 1.0f;
  float u[3], v[3];
  for (int k = 0; k < 3; ++k) {
    u[k] = cv[k].c[0] - pxn * cv[k].c[3];
    v[k] = cv[k].c[1] - pyn * cv[k].c[3];
  }
  float b0 = u[1] * v[2] - u[2] * v[1], b1 = u[2] * v[0] - u[0] * v[2], b2 = u[0] * v[1] - u[1] * v[0];
  const float sb = b0 + b1 + b2;
  if (sb != 0.0f) {
    const float inv = 1.0f / sb;
    b0 *= inv; b1 *= inv; b2 *= inv;
  } else {
    b0 = b1 = b2 = 1.0f / 3.0f;
  }
  const V3 world = wp[0] * b0 + wp[1] * b1 + wp[2] * b2;
  const V3 nrm = nn[0] * b0 + nn[1] * b1 + nn[2] * b2;
  const uint32_t mat = __ldg(sp.obj_material + __ldg(in.tri_obj + lt));
  rb.gb_pos[p] = make_float4(world.x, world.y, world.z, __uint_as_float(mat));
  rb.gb_nrm[p] = make_float4(nrm.x, nrm.y, nrm.z, __uint_as_float(t));
}

__global__ void __launch_bounds__(256) k_gb_resolve(SceneParams sp, CameraParams cp, RasterBuffers rb) {
  follows_previous();
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *rb.big_count = 0;  // for the next frame
  resolve_px(sp, cp, rb, blockIdx.x * 16 + (threadIdx.x & 15), blockIdx.y * 16 + (threadIdx.x >> 4));
}

// 16x16-pixel tiles of every batch scene.
__global__ void __launch_bounds__(256) k_gb_resolve_batch(BatchWork w, RasterBuffers rb) {
  follows_previous();
  if (blockIdx.x == 0 && threadIdx.x == 0) *rb.big_count = 0;  // for the next frame
  for (uint32_t g = blockIdx.x; g < w.total; g += gridDim.x) {
    const int s = batch_scene_of(w, g);
    const BatchScene& S = w.scenes[s];
    const uint32_t lt = g - __ldg(w.prefix + s), tiles_x = (uint32_t)(S.W + 15) / 16;
    resolve_px(S.sp, w.cams[s], scene_rb(rb, S), (int)(lt % tiles_x) * 16 + (threadIdx.x & 15),
               (int)(lt / tiles_x) * 16 + (threadIdx.x >> 4));
  }
}

}  // namespace

size_t big_record_bytes() { return sizeof(BigRec); }

cudaError_t launch_gbuffer(const SceneParams& sp, const CameraParams& cp, const RasterBuffers& rb, cudaStream_t st,
                           int* launches) {
  cudaError_t e = cudaMemsetAsync(rb.vis, 0xff, (size_t)cp.W * cp.H * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  if (sp.total_tris) {
    auto setup = snap_wide(cp.W, cp.H) ? k_gb_setup<true> : k_gb_setup<false>;
    setup<<<(sp.total_tris + kSetup - 1) / kSetup, kSetup, 0, st>>>(sp, cp, rb);
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  e = launch_next(k_gb_big, sms * 6, 256, st, rb, cp.W, nullptr);
  if (e != cudaSuccess) return e;
  dim3 grid((cp.W + 15) / 16, (cp.H + 15) / 16);
  e = launch_next(k_gb_resolve, grid, 256, st, sp, cp, rb);
  if (e != cudaSuccess) return e;
  if (launches) *launches += (sp.total_tris ? 1 : 0) + 2;
  return cudaGetLastError();
}

cudaError_t launch_gbuffer_batch(const BatchWork& tris, const BatchWork& tiles, size_t total_px,
                                 const BatchBuffers& bb, int sms, cudaStream_t st, int* launches) {
  const RasterBuffers& rb = bb.rb;
  cudaError_t e = cudaMemsetAsync(rb.vis, 0xff, total_px * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  int nl = 0;
  if (tris.total) {
    const unsigned grid = (unsigned)std::max(1, std::min<int>(sms * 32, (int)((tris.total + kSetup - 1) / kSetup)));
    k_gb_setup_batch<<<grid, kSetup, 0, st>>>(tris, rb);
    ++nl;
  }
  e = launch_next(k_gb_big, sms * 6, 256, st, rb, 0, tris.scenes);
  if (e != cudaSuccess) return e;
  const unsigned rgrid = (unsigned)std::max(1, std::min<int>(sms * 8, (int)tiles.total));
  e = launch_next(k_gb_resolve_batch, rgrid, 256, st, tiles, rb);
  if (e != cudaSuccess) return e;
  nl += 2;
  if (launches) *launches += nl;
  return cudaGetLastError();
}

}  // namespace vct
