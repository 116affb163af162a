// Host check of rayorder.hpp over the fake runtime (fake_cuda.hpp): a sequence
// of uses of growing size on a device with and without room, with a failure at
// every call and at every launch. Whenever the kernels are launched, the arrays
// hold the slots asked for and the counts are zero; a failure leaves nothing
// that a later, sound use could trip over; freeing leaves nothing behind.
// Prints the cases checked.
#include <cstdio>
#include <initializer_list>

#include "fake_cuda.hpp"

#include "../myrt_b200/csrc/rayorder.hpp"

using namespace myrt_b200;

static bool sound = true;
static void check(bool ok, char const* what) {
  if (!ok) std::printf("%s\n", what);
  sound = sound && ok;
}

// The arrays lie side by side in the two allocations, each as long as its use of n slots needs.
static void check_layout(ray_order const& o, size_t n) {
  auto at = [](void const* p) { return reinterpret_cast<uintptr_t>(p); };
  size_t const warps = (n + 31) / 32;
  check(o.cap >= n, "fewer slots than asked for");
  check(at(o.dev.count) == at(o.cells) && at(o.dev.offset) >= at(o.dev.count) + 4 * size_t(kOrderBins) &&
            at(o.dev.ctr) >= at(o.dev.offset) + 4 * size_t(kOrderBins) &&
            at(o.cells) + fake::memory.at(o.cells) >= at(o.dev.ctr) + 16, "cells' tables");
  check(at(o.dev.rec) == at(o.slots) && at(o.dev.perm) >= at(o.dev.rec) + 8 * 32 * warps &&
            at(o.dev.warp) >= at(o.dev.perm) + 4 * 32 * warps &&
            at(o.slots) + fake::memory.at(o.slots) >= at(o.dev.warp) + 4 * warps, "slots' arrays");
  // k_order_offsets reads and writes 16 bytes at a time
  check(at(o.dev.count) % 16 == 0 && at(o.dev.offset) % 16 == 0, "alignment");
}

// One use of n slots as the library makes it; bad_launch: the kernels after the
// count do not start, so the counts stay.
static bool use(ray_order& o, size_t n, bool bad_launch) {
  cudaStream_t const s = fake::stream(1);
  bool const fits = o.cap >= n && o.clean;
  int const before = fake::calls;
  cudaError_t e = ensure_ray_order(o, n, s);
  check(!fits || fake::calls == before, "calls without need");
  check((e != cudaSuccess) == (!fits && fake::fail_at == before), "a failed wait hidden, or an error without one");
  check(fake::last == cudaSuccess, "an error left for the next launch check");
  if (e != cudaSuccess) return false;
  if (o.cap < n) {
    check(o.cap == 0 && fake::held == 0, "no room, but memory held");
    return false;
  }
  e = use_ray_order(o, s, [&] {
    bool zero = true;
    for (size_t i = 0; i < kOrderBins; i += 61) zero = zero && o.dev.count[i] == 0;
    check(zero, "counts left behind");
    check_layout(o, n);
    check(o.dev.ctr[0] == 0 && o.dev.ctr[1] == 0 && o.dev.ctr[2] == 0, "counters not zero");
    if (bad_launch) {
      for (size_t i = 0; i < kOrderBins; i += 61) o.dev.count[i] = 7;
      fake::last = cudaErrorLaunchOutOfResources;
    }
  });
  return e == cudaSuccess;
}

// Queries on two streams that share one scratch as api.cu's launch_trace does:
// each waits for the one before, also when that one's traversal launch failed.
static void shared(int bad) {
  cudaEvent_t const done = fake::event(9);
  ray_order o;
  std::set<int> users;
  for (int k = 0; k < 6; ++k) {
    cudaStream_t const s = fake::stream(1 + k % 2);
    if (cudaStreamWaitEvent(s, done, 0) != cudaSuccess) continue;
    bool used = false;
    if (ensure_ray_order(o, 100, s) == cudaSuccess && o.cap >= 100) {
      used = true;
      use_ray_order(o, s, [&] {
        for (int w : users) check(fake::after[s].count(w) || fake::host.count(w), "a use beside another");
        users.insert(fake::launch(s));
      });
    }
    bool const traversal_failed = k == bad;
    if (!traversal_failed && used) users.insert(fake::launch(s));
    if (used) mark_ray_order_use(done, s);
  }
  fake::last = cudaSuccess;
  free_ray_order(o);
}

int main() {
  int checked = 0;
  for (int bad = -1; bad < 6; ++bad)
    for (int fail = -1; fail < 32; ++fail) {
      fake::reset(fail);
      shared(bad);
      if (!sound) {
        std::printf("shared: bad traversal %d, failing call %d\n", bad, fail);
        return 1;
      }
      ++checked;
    }
  for (size_t limit : {SIZE_MAX, size_t(34) << 20, size_t(16) << 20})
    for (int bad = -1; bad < 3; ++bad)
      for (int fail = -1; fail < 24; ++fail) {
        fake::reset(fail);
        fake::limit = limit;
        ray_order o;
        int k = 0, done = 0;
        for (size_t n : {40, 1000, 1000, 70000, 33})
          done += use(o, n, k++ == bad);
        fake::limit = SIZE_MAX;
        fake::fail_at = -1;
        check(use(o, 50000, false), "no recovery");
        if (limit == SIZE_MAX && bad < 0 && fail < 0)
          check(done == 5 && fake::mallocs == 4 && fake::frees == 2, "sound uses: one table, a slots' part per growth");
        free_ray_order(o);
        check(fake::held == 0, "memory left");
        if (!sound) {
          std::printf("limit %zu, bad launch %d, failing call %d\n", limit, bad, fail);
          return 1;
        }
        ++checked;
      }
  std::printf("%d\n", checked);
  return 0;
}
