// Host check of call_buffer.hpp over the fake runtime (fake_cuda.hpp): calls on
// host arrays of several sizes -- take, upload, kernels, read back, wait, end --
// with a failure at every call they make. When a call returns, nothing of it is
// still running, a sound call has its buffer, and no more than the kept size
// stays held. Prints the cases checked.
#include <cstdio>
#include <initializer_list>

#include "fake_cuda.hpp"

#include "../myrt_b200/csrc/call_buffer.hpp"

static cudaError_t async(cudaStream_t s) {  // a copy or a launch
  if (fake::fails()) return cudaErrorUnknown;
  fake::launch(s);
  return cudaSuccess;
}

int main() {
  int checked = 0;
  for (int fail = -1; fail < 32; ++fail) {
    fake::reset(fail);
    cudaStream_t const s = fake::stream(1);
    myrt_b200::call_buffer b;
    bool sound = true;
    int failed = 0;
    for (size_t bytes : {size_t(1) << 10, size_t(70) << 20, size_t(64) << 20, size_t(1) << 10}) {
      cudaError_t e = b.take(bytes);
      if (e == cudaSuccess) {
        sound = sound && b.cap >= bytes && fake::memory.at(b.p) >= bytes;
        for (int k = 0; k < 4 && e == cudaSuccess; ++k) e = async(s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        b.end_call(s, e != cudaSuccess);
      }
      failed += e != cudaSuccess;
      for (int w : fake::after[s]) sound = sound && fake::host.count(w);
      sound = sound && fake::held == b.cap && b.cap <= myrt_b200::call_buffer::kKeep;
    }
    sound = sound && failed == (fail >= 0 && fail < fake::calls);
    b.free();
    if (!sound || fake::held) {
      std::printf("failing call %d\n", fail);
      return 1;
    }
    ++checked;
  }
  std::printf("%d\n", checked);
  return 0;
}
