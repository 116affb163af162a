// Host side of a visiting order's scratch (rayorder.cuh): its arrays, and what
// holds between uses.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime_api.h>

namespace myrt_b200 {

constexpr uint32_t kOrderCells = 1u << 22;
constexpr uint32_t kOrderChunk = 4096;                       // cells per block of k_order_offsets
constexpr uint32_t kOrderBins = kOrderCells + kOrderChunk;   // and the cell of empty slots

// 12 bytes per slot and 32 MB.
struct ray_order_dev {
  uint32_t* count = nullptr;   // rays per cell, zero between uses
  uint32_t* offset = nullptr;  // first position of a cell's rays
  uint2* rec = nullptr;        // (cell, rank) of every ray of the warps taken apart
  uint32_t* warp = nullptr;    // those warps' first slots
  uint32_t* perm = nullptr;    // the order: slot of the i-th thread
  uint32_t* ctr = nullptr;     // warps taken apart, rays of the others, positions given out
};
// Two allocations, the cells' tables kept while the slots' part grows: a cudaMalloc costs the first
// query of a context 0.3 ms whatever its size (and tens of ms when the host is busy). First query of
// 1 Mi / 28 M rays, and 28 M after 1 Mi: six allocations 1.75 / 7.7 / 9.0 ms, two 1.15 / 6.7 / 6.7 ms
// (the radix sort's five: 2.2 / 8.4 / 10.2).
struct ray_order {
  ray_order_dev dev;   // count, offset and ctr in `cells`; rec, perm and warp in `slots`
  void* cells = nullptr;
  void* slots = nullptr;
  size_t cap = 0;      // slots
  bool clean = false;  // the counts are zero; not after a use whose launches may have run in part
};

inline void free_ray_order(ray_order& o) {
  cudaFree(o.cells);
  cudaFree(o.slots);
  o = ray_order{};
}

// Room for n slots, with zero counts, where the device has it; without it
// nothing is held, o.cap is below n and the caller visits in input order. An
// error is a stream that cannot be waited for: work before it failed, or it is
// being captured, when no memory may be taken.
inline cudaError_t ensure_ray_order(ray_order& o, size_t n, cudaStream_t s) {
  if (o.cap >= n && o.clean) return cudaSuccess;
  if (cudaError_t const e = cudaStreamSynchronize(s); e != cudaSuccess) {
    cudaGetLastError();
    return e;
  }
  if (o.cap < n) {
    size_t const bins = kOrderBins, warps = (n + 31) / 32;
    cudaFree(o.slots);
    o.slots = nullptr;
    o.cap = 0;
    if ((o.cells || cudaMalloc(&o.cells, (2 * bins + 4) * 4) == cudaSuccess) &&
        cudaMalloc(&o.slots, warps * (32 * 12 + 4)) == cudaSuccess) {
      auto* const c = static_cast<uint32_t*>(o.cells);
      auto* const rec = static_cast<uint2*>(o.slots);
      auto* const perm = reinterpret_cast<uint32_t*>(rec + warps * 32);
      o.dev = ray_order_dev{c, c + bins, rec, perm + warps * 32, perm, c + 2 * bins};
      o.cap = n;
    }
  }
  o.clean = o.cap >= n && cudaMemsetAsync(o.dev.count, 0, size_t(kOrderBins) * 4, s) == cudaSuccess;
  if (!o.clean) {
    cudaGetLastError();
    free_ray_order(o);
  }
  return cudaSuccess;
}

// One use: launch() starts the kernels that count, turn counts into positions
// (zeroing them again) and scatter. Counts that a failed launch leaves behind
// would push a later use's positions past the order's end, so the scratch is
// then unfit until ensure_ray_order has cleared it.
template <class LAUNCH>
cudaError_t use_ray_order(ray_order& o, cudaStream_t s, LAUNCH const& launch) {
  o.clean = false;
  cudaError_t const e = cudaMemsetAsync(o.dev.ctr, 0, 4 * sizeof(uint32_t), s);
  if (e == cudaSuccess) launch();
  cudaError_t const l = cudaGetLastError();  // also takes back the clearing's own error
  o.clean = e == cudaSuccess && l == cudaSuccess;
  return e != cudaSuccess ? e : l;
}

// Records the end of a use for the streams of later uses; where that fails, the
// host waits for it instead.
inline cudaError_t mark_ray_order_use(cudaEvent_t done, cudaStream_t s) {
  cudaError_t const e = cudaEventRecord(done, s);
  if (e != cudaSuccess) cudaStreamSynchronize(s);
  return e;
}

}  // namespace myrt_b200
