// Host check of stream_fork.hpp over the fake runtime (fake_cuda.hpp): a chain
// like a path wave's -- work on a stream, a fork, the next work beside it, a
// join -- left by an error at every call it makes, and by an error of its own
// between fork and join. However it is left, the first stream or the host has
// waited for everything launched on the second. Prints the cases checked.
#include <cstdio>

#include "fake_cuda.hpp"

#include "../myrt_b200/csrc/stream_fork.hpp"

// step: where the chain returns by itself (-1: never), counted over its points
static cudaError_t chain(int step, bool& ordered) {
  cudaStream_t const main_s = fake::stream(1), side_s = fake::stream(2);
  myrt_b200::stream_fork side(main_s, side_s, fake::event(3), fake::event(4));
  int at = 0;
  std::set<int> beside;
  for (int v = 0; v < 3; ++v) {
    fake::launch(main_s);  // extension, beside the shadow rays of the vertex before
    if (at++ == step) return cudaErrorUnknown;
    if (cudaError_t const e = side.join()) return e;
    for (int w : beside) ordered = ordered && fake::after[main_s].count(w);
    int const shade = fake::launch(main_s);
    if (cudaError_t const e = side.fork()) return e;
    if (at++ == step) return cudaErrorUnknown;
    ordered = ordered && fake::after[side_s].count(shade);
    beside.insert(fake::launch(side_s));
    if (at++ == step) return cudaErrorUnknown;
    if (cudaError_t const e = side.launched()) return e;
  }
  return side.join();
}

int main() {
  int checked = 0;
  for (int step = -1; step < 9; ++step)
    for (int fail = -1; fail < 32; ++fail) {
      fake::reset(fail);
      bool ordered = true;
      cudaError_t const e = chain(step, ordered);
      bool const want_error = step >= 0 || (fail >= 0 && fail < fake::calls);
      bool waited = true;
      for (int w : fake::after[fake::stream(2)])
        waited = waited && (fake::after[fake::stream(1)].count(w) || fake::host.count(w));
      if (!ordered || !waited || (e != cudaSuccess) != want_error) {
        std::printf("step %d, failing call %d: ordered %d, waited %d, error %d\n", step, fail, ordered, waited, int(e));
        return 1;
      }
      ++checked;
    }
  std::printf("%d\n", checked);
  return 0;
}
