// Device memory for one call on host arrays, kept between calls: cudaMalloc and
// the synchronising cudaFree of two buffers cost a guide evaluation or training
// call about as much as its kernels. Calls of one context run one after another
// on its stream.
#pragma once
#include <cstddef>
#include <cuda_runtime_api.h>

namespace myrt_b200 {

struct call_buffer {
  static constexpr size_t kKeep = size_t(64) << 20;  // larger buffers go back at the end of their call
  void* p = nullptr;
  size_t cap = 0;

  void free() {
    cudaFree(p);
    p = nullptr;
    cap = 0;
  }
  cudaError_t take(size_t bytes) {
    if (cap >= bytes) return cudaSuccess;
    free();
    cudaError_t const e = cudaMalloc(&p, bytes);
    if (e == cudaSuccess) cap = bytes;
    else p = nullptr;
    return e;
  }
  // The end of a call. One that failed has not waited for its stream: copies from and to the
  // caller's arrays may be under way, and the arrays are the caller's again once it returns.
  void end_call(cudaStream_t s, bool failed) {
    if (failed) cudaStreamSynchronize(s);
    if (cap > kKeep) free();
  }
};

}  // namespace myrt_b200
