// A fake of the few CUDA runtime calls that the library's host-side helpers
// make, for checks without a GPU: streams and events carry the set of work
// they are ordered after, memory comes from the heap up to a limit, and the
// call numbered `fail_at` (from 0) fails without effect.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <vector>

namespace fake {

inline std::map<void const*, std::set<int>> after;  // stream or event -> work it is ordered after
inline std::set<int> host;                          // work the host has waited for
inline int launched = 0, calls = 0, fail_at = -1;
inline cudaError_t fail_with = cudaErrorUnknown, last = cudaSuccess;
inline std::map<void*, std::size_t> memory;         // live allocations
inline std::size_t held = 0, limit = SIZE_MAX;
inline int mallocs = 0, frees = 0;

inline void reset(int fail) {
  for (auto& m : memory) std::free(m.first);
  memory.clear();
  after.clear();
  host.clear();
  launched = calls = mallocs = frees = 0;
  held = 0;
  limit = SIZE_MAX;
  fail_at = fail;
  last = cudaSuccess;
}
inline bool fails() { return calls++ == fail_at; }
inline cudaError_t result(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
inline cudaStream_t stream(std::uintptr_t k) { return reinterpret_cast<cudaStream_t>(16 * k); }
inline cudaEvent_t event(std::uintptr_t k) { return reinterpret_cast<cudaEvent_t>(16 * k + 8); }
inline int launch(cudaStream_t s) {
  after[s].insert(launched);
  return launched++;
}

}  // namespace fake

extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  if (fake::fails()) return fake::result(fake::fail_with);
  fake::after[e] = fake::after[s];
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (fake::fails()) return fake::result(fake::fail_with);
  fake::after[s].insert(fake::after[e].begin(), fake::after[e].end());
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (fake::fails()) return fake::result(fake::fail_with);
  fake::host.insert(fake::after[s].begin(), fake::after[s].end());
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes) {
  if (fake::fails()) return fake::result(fake::fail_with);
  if (fake::held + bytes > fake::limit) return fake::result(cudaErrorMemoryAllocation);
  *p = std::malloc(bytes ? bytes : 1);
  std::memset(*p, 0xab, bytes);
  fake::memory[*p] = bytes;
  fake::held += bytes;
  ++fake::mallocs;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  fake::held -= fake::memory.at(p);
  fake::memory.erase(p);
  std::free(p);
  ++fake::frees;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t) {
  if (fake::fails()) return fake::result(fake::fail_with);
  std::memset(p, v, bytes);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  cudaError_t const e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
}
