// Visiting order of a batch of rays. Rays are grouped by a 22-bit cell: the
// Morton code of the origin's cell in a 16^3 grid over the scene box, then the
// Morton code of the direction's cell in a 32^2 octahedral grid. Neighbouring
// lanes of a warp then walk similar paths through the tree (fewer divergent
// branches, node and triangle loads shared through L1). Every result is written
// at its ray's own index, so the order never changes any answer.
//
// Only warps that gain from it are taken apart: 32 neighbouring rays that lie in
// at most kCoherentCells cells (camera rays, image rows) stay together and go
// first; the others are counting-sorted by cell. Three kernels:
//   k_order_cells    cell of every ray; whole coherent warps straight into the
//                    order, the rays of the others counted per cell, the count
//                    before being the ray's rank
//   k_order_offsets  counts -> first positions (and the counts back to zero)
//   k_order_scatter  rays to first position + rank
// Cells come in order within 4,096 of them; which of those chunks comes first,
// and the rays' order inside a cell, follow the blocks' arrival. Measured by
// sorting rays on the same keys (traversal alone, 27.9 M closest hits): arrival
// order 6.27 ms, a stable order 6.18 ms; camera rays kept out, as all 16^3 x 16^3
// cells (24 bits) in the same order 6.26 ms, 18 bits 6.71 ms.
//
// Cost against the radix sort of (24-bit key, index) pairs that stood here:
// 2^20 camera rays 58 -> 17 us, 27.9 M rays (60 % of them camera rays) 840 ->
// 354 us, of which 150 us is reading the rays.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "rayorder.hpp"

namespace myrt_b200 {

// Batches from this size on are ordered (trace_order 0).
constexpr uint32_t kOrderMin = 1u << 20;
constexpr uint32_t kOrderTile = 1024;                        // rays per block of k_order_cells
constexpr uint32_t kOrderScatterBlocks = 148 * 8;            // one resident wave, however few warps were taken apart
// Camera rays of a 1024 x 1024 image lie in 1.3 cells per warp, of a 512 x 512 one in 1.5, shadow
// rays of neighbouring hits in 24 and bounce rays in 32: 4, 8 and 12 measured the same.
constexpr int kCoherentCells = 8;

__device__ __forceinline__ uint32_t spread4(uint32_t v) {  // the low 4 bits of v to bits 0, 3, 6, 9
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}
__device__ __forceinline__ uint32_t spread5(uint32_t v) {  // the low 5 bits of v to bits 0, 2, 4, 6, 8
  return (v & 1u) | ((v & 2u) << 1) | ((v & 4u) << 2) | ((v & 8u) << 3) | ((v & 16u) << 4);
}
__device__ __forceinline__ uint32_t order_cell(float x, float last) {  // 0 .. last, clamped (NaN -> 0)
  return x >= last ? uint32_t(last) : (x > 0.f ? uint32_t(x) : 0u);
}

// The cell of a ray with origin o and direction d (any length); lo and
// cell_scale map the scene box onto [0, 16)^3.
__device__ __forceinline__ uint32_t ray_cell(float4 o, float4 d, float3 lo, float3 cell_scale) {
  uint32_t const ox = order_cell((o.x - lo.x) * cell_scale.x, 15.f);
  uint32_t const oy = order_cell((o.y - lo.y) * cell_scale.y, 15.f);
  uint32_t const oz = order_cell((o.z - lo.z) * cell_scale.z, 15.f);
  float const l1 = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
  float const s = l1 > 0.f ? __fdividef(1.f, l1) : 0.f;
  float px = d.x * s, py = d.y * s;
  if (d.z < 0.f) {
    float const qx = copysignf(1.f - fabsf(py), px);
    py = copysignf(1.f - fabsf(px), py);
    px = qx;
  }
  uint32_t const u = order_cell(fmaf(px, 16.f, 16.f), 31.f), v = order_cell(fmaf(py, 16.f, 16.f), 31.f);
  uint32_t const om = spread4(ox) | (spread4(oy) << 1) | (spread4(oz) << 2);
  return (om << 10) | spread5(u) | (spread5(v) << 1);
}

// cell_of(i): the cell of slot i < n, kOrderCells when it holds no ray.
// n_dev (may be null): the number of slots, at most n, on the device.
// ctr[0]: the warps taken apart, ctr[1]: the rays of the others, ctr[2]: for
// k_order_offsets; zero at the start, like every count.
template <class CELL>
static __global__ void __launch_bounds__(256) k_order_cells(CELL cell_of, uint32_t n,
    uint32_t const* __restrict__ n_dev, ray_order_dev r) {
  __shared__ uint32_t split, first_split, first_whole;
  if (n_dev) n = min(n, *n_dev);
  uint32_t const base = blockIdx.x * kOrderTile;
  if (base >= n) return;
  uint32_t const lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, rays = min(kOrderTile, n - base);
  if (threadIdx.x == 0) split = 0;
  __syncthreads();
  uint32_t cell[4], peers[4];
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    uint32_t const at = (warp * 4 + k) * 32 + lane;
    cell[k] = at < rays ? cell_of(base + at) : kOrderCells;
  }
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    peers[k] = __match_any_sync(0xffffffffu, cell[k]);
    bool const leader = lane == uint32_t(__ffs(int(peers[k]))) - 1u;
    int const cells = __popc(__ballot_sync(0xffffffffu, leader));
    // the last, partial warp stays whole: the warps taken apart hold 32 rays each
    if (lane == 0 && cells > kCoherentCells && (warp * 4 + k) * 32 + 32 <= rays)
      atomicOr(&split, 1u << (warp * 4 + k));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t const parts = uint32_t(__popc(split)), whole = rays - 32u * parts;
    if (parts) first_split = atomicAdd(r.ctr, parts);
    if (whole) first_whole = atomicAdd(r.ctr + 1, whole);
  }
  __syncthreads();
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    uint32_t const t = warp * 4 + k, at = t * 32 + lane, before = uint32_t(__popc(split & ((1u << t) - 1u)));
    if (split >> t & 1u) {
      uint32_t const leader = uint32_t(__ffs(int(peers[k]))) - 1u;
      uint32_t rank = 0;
      if (lane == leader) rank = atomicAdd(r.count + cell[k], uint32_t(__popc(peers[k])));
      rank = __shfl_sync(0xffffffffu, rank, int(leader)) + uint32_t(__popc(peers[k] & ((1u << lane) - 1u)));
      uint32_t const slot = first_split + before;
      r.rec[size_t(slot) * 32 + lane] = make_uint2(cell[k], rank);
      if (lane == 0) r.warp[slot] = base + t * 32;
    } else if (at < rays) {
      r.perm[first_whole + (t - before) * 32 + lane] = base + at;
    }
  }
}

static __global__ void __launch_bounds__(1024) k_order_offsets(ray_order_dev r) {
  __shared__ uint32_t warp_sum[32], start;
  if (r.ctr[0] == 0) return;  // every warp stayed whole: all counts are zero
  uint32_t const lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t const i = blockIdx.x * (kOrderChunk / 4) + threadIdx.x;
  uint4 const c = reinterpret_cast<uint4 const*>(r.count)[i];
  uint32_t const sum = c.x + c.y + c.z + c.w;
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t const y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= uint32_t(o)) x += y;
  }
  if (lane == 31) warp_sum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t const own = warp_sum[lane];
    uint32_t w = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t const y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= uint32_t(o)) w += y;
    }
    warp_sum[lane] = w - own;
    if (lane == 31 && w) start = atomicAdd(r.ctr + 2, w);
  }
  __syncthreads();
  if (sum == 0) return;
  uint32_t const at = start + warp_sum[warp] + x - sum;
  reinterpret_cast<uint4*>(r.offset)[i] = make_uint4(at, at + c.x, at + c.x + c.y, at + c.x + c.y + c.z);
  reinterpret_cast<uint4*>(r.count)[i] = make_uint4(0, 0, 0, 0);
}

static __global__ void __launch_bounds__(256) k_order_scatter(uint32_t n, uint32_t const* __restrict__ n_dev,
    ray_order_dev r) {
  uint32_t const lane = threadIdx.x & 31u, parts = r.ctr[0];
  if (n_dev) n = min(n, *n_dev);
  for (uint32_t slot = blockIdx.x * 8 + (threadIdx.x >> 5); slot < parts; slot += gridDim.x * 8) {
    uint2 const e = r.rec[size_t(slot) * 32 + lane];
    r.perm[n - parts * 32 + r.offset[e.x] + e.y] = r.warp[slot] + lane;
  }
}

// The scene box [b[0..2], b[3..5]] -> lo and cell_scale of ray_cell.
inline void ray_cell_grid(float const* b, float3& lo, float3& cell_scale) {
  float* plo = &lo.x;
  float* psc = &cell_scale.x;
  for (int k = 0; k < 3; ++k) {
    float const ext = b[3 + k] - b[k];
    plo[k] = b[k] - 1e-3f * ext;
    psc[k] = ext > 0.f ? 16.f / (ext * 1.002f) : 0.f;
  }
}

// The order of n slots into o.dev.perm (room for them made before).
template <class CELL>
cudaError_t build_ray_order(ray_order& o, CELL const& cell_of, uint32_t n, uint32_t const* n_dev, cudaStream_t s) {
  return use_ray_order(o, s, [&] {
    ray_order_dev const r = o.dev;
    k_order_cells<<<uint32_t((size_t(n) + kOrderTile - 1) / kOrderTile), 256, 0, s>>>(cell_of, n, n_dev, r);
    k_order_offsets<<<kOrderBins / kOrderChunk, kOrderChunk / 4, 0, s>>>(r);
    k_order_scatter<<<std::min(kOrderScatterBlocks, uint32_t((size_t(n) + 255) / 256)), 256, 0, s>>>(n, n_dev, r);
  });
}

}  // namespace myrt_b200
