// Work beside a stream: launches on a second stream that begin after what the
// first holds so far and that the first waits for at join().
//
// A caller that leaves early -- an error between the fork and the join -- must
// not leave the second stream running: the buffers belong to the next call by
// then, nobody waits for that stream, and a capture would end unjoined. So the
// destructor joins too, and a join that cannot be recorded waits on the host.
#pragma once
#include <cuda_runtime_api.h>

namespace myrt_b200 {

class stream_fork {
public:
  // forked, joined: two events of the caller's, one fork at a time
  stream_fork(cudaStream_t main, cudaStream_t side, cudaEvent_t forked, cudaEvent_t joined)
      : main_(main), side_(side), forked_(forked), joined_(joined) {}
  stream_fork(stream_fork const&) = delete;
  stream_fork& operator=(stream_fork const&) = delete;
  ~stream_fork() { join(); }

  // The second stream waits for what the first holds; launches go there until launched().
  cudaError_t fork() {
    cudaError_t e = cudaEventRecord(forked_, main_);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side_, forked_, 0);
    if (e != cudaSuccess) return e;
    open_ = true;
    recorded_ = false;
    return cudaSuccess;
  }
  // Marks the end of the fork's launches.
  cudaError_t launched() {
    cudaError_t const e = cudaEventRecord(joined_, side_);
    recorded_ = e == cudaSuccess;
    return e;
  }
  // The first stream waits for the fork's launches; nothing to do without a fork.
  cudaError_t join() {
    if (!open_) return cudaSuccess;
    open_ = false;
    cudaError_t e = recorded_ ? cudaSuccess : launched();
    if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, joined_, 0);
    if (e != cudaSuccess) cudaStreamSynchronize(side_);
    return e;
  }

private:
  cudaStream_t main_, side_;
  cudaEvent_t forked_, joined_;
  bool open_ = false, recorded_ = false;
};

}  // namespace myrt_b200
