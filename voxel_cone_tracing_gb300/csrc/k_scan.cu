// k_scan.cu -- device-wide exclusive prefix sum of u32 counts (brick list
// offsets of the voxelizer): a scan per tile, then the add-back, whose CTAs
// sum the tile totals for themselves.
#include <cstring>

#include "vct_internal.h"

namespace vct {
namespace {

constexpr int kT = 1024;          // threads per tile
constexpr int kI = 4;             // items per thread
constexpr int kTile = kT * kI;

// Exclusive block scan of one value per thread; returns the block total.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t& excl) {
  __shared__ uint32_t warp_tot[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0u;
    uint32_t wi = w;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_tot[lane] = wi - w;  // exclusive warp offsets
  }
  __syncthreads();
  excl = warp_tot[warp] + incl - v;
  uint32_t total = __shfl_sync(0xffffffffu, incl, 31) + warp_tot[warp];
  total = __shfl_sync(0xffffffffu, total, 31);
  __shared__ uint32_t s_total;
  if (threadIdx.x == blockDim.x - 1) s_total = excl + v;
  __syncthreads();
  uint32_t r = s_total;
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kT) k_scan_tiles(const uint32_t* in, uint32_t* __restrict__ out,
                                                   uint32_t* __restrict__ tile_tot, size_t n, ScanFuse fuse) {
  follows_previous();
  if (blockIdx.x == 0) {  // the counters of the plan and of the list, before k_scan_add
    if (fuse.hb.slot && threadIdx.x < 2) fuse.hb.counters[threadIdx.x] = 0u;
    if (fuse.units.list && threadIdx.x < 3) fuse.units.count[threadIdx.x] = 0u;
  }
  const size_t base = (size_t)blockIdx.x * kTile + (size_t)threadIdx.x * kI;
  uint32_t v[kI];
  uint32_t s = 0;
  for (int i = 0; i < kI; ++i) {
    v[i] = base + i < n ? in[base + i] : 0u;
    s += v[i];
  }
  uint32_t ex;
  const uint32_t tot = block_excl_scan(s, ex);
  for (int i = 0; i < kI; ++i) {
    if (base + i < n) out[base + i] = ex;
    ex += v[i];
  }
  if (threadIdx.x == 0) tile_tot[blockIdx.x] = tot;
}

// Adds each tile the totals of those before it (every CTA sums them itself:
// at most a few hundred words, against a launch of its own), and plans the
// bricks.
__global__ void __launch_bounds__(256) k_scan_add(uint32_t* in, uint32_t* out,
                                                  uint32_t* __restrict__ copy_out,
                                                  const uint32_t* tile_tot, uint32_t ntiles, size_t n,
                                                  ScanFuse fuse) {
  follows_previous();
  __shared__ uint32_t s_before[8], s_all[8];
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t tile = (uint32_t)((size_t)blockIdx.x * blockDim.x / kTile);  // one for the whole CTA
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t before = 0, all = 0;
  for (uint32_t k = threadIdx.x; k < ntiles; k += 256) {
    const uint32_t v = tile_tot[k];
    all += v;
    before += k < tile ? v : 0u;
  }
  before = __reduce_add_sync(0xffffffffu, before);
  all = __reduce_add_sync(0xffffffffu, all);
  if (lane == 0) {
    s_before[warp] = before;
    s_all[warp] = all;
  }
  __syncthreads();
  before = all = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    before += s_before[w];
    all += s_all[w];
  }
  if (i == 0) {
    out[n] = all;
    if (fuse.total_copy) *fuse.total_copy = all;
    if (fuse.big_total) *fuse.big_total = *fuse.big_count;
  }
  const uint32_t c = fuse.cap;
  uint32_t pairs = 0;
  if (i < n) {
    const uint32_t v = out[i] + before, cnt = in[i];
    out[i] = v;
    if (copy_out) copy_out[i] = v;
    if (fuse.clear) in[i] = 0u;
    if (fuse.hb.slot) heavy_plan_brick((uint32_t)i, min(v, c), min(v + cnt, c), min(all, c), fuse.slots, fuse.hb);
    pairs = min(v + cnt, c) - min(v, c);
  }
  if (!fuse.units.list) return;
  const BrickUnits& u = fuse.units;
  const int kind = i >= n ? 2 : pairs > kLongBrick ? 0 : pairs || !u.dirty || u.dirty[i] ? 1 : 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const unsigned m = __ballot_sync(0xffffffffu, kind == k);
    if (!m) continue;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&u.count[k], (uint32_t)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (kind == k) u.list[k ? u.cap - 1u - at : at] = (uint32_t)i;
  }
}

}  // namespace

size_t scan_tmp_words(size_t n) { return (n + kTile - 1) / kTile + 1; }

cudaError_t launch_exclusive_scan(uint32_t* in, uint32_t* out, uint32_t* copy_out, size_t n, uint32_t* tmp,
                                  cudaStream_t st, int* launches, const ScanFuse* fuse) {
  ScanFuse f;
  std::memset(&f, 0, sizeof(f));
  if (fuse) f = *fuse;
  if (n == 0) {
    // No bricks: nothing to plan (the counters still start at zero).
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess && f.total_copy) e = cudaMemsetAsync(f.total_copy, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess && f.hb.slot) e = cudaMemsetAsync(f.hb.counters, 0, 2 * sizeof(uint32_t), st);
    if (e == cudaSuccess && f.units.list) e = cudaMemsetAsync(f.units.count, 0, 3 * sizeof(uint32_t), st);
    return e;
  }
  const size_t ntiles = (n + kTile - 1) / kTile;
  cudaError_t e = launch_next(k_scan_tiles, (unsigned)ntiles, kT, st, in, out, tmp, n, f);
  if (e != cudaSuccess) return e;
  e = launch_next(k_scan_add, (unsigned)((n + 255) / 256), 256, st, in, out, copy_out, tmp, (uint32_t)ntiles, n, f);
  if (e != cudaSuccess) return e;
  if (launches) *launches += 2;
  return cudaGetLastError();
}

}  // namespace vct
