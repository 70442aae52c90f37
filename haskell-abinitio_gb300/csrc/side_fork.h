// Work on side streams between a fork from and a join into a context's stream.
#pragma once
#include <cuda_runtime.h>

namespace gbhf {

// fork(): the n side streams wait for what the main stream holds so far; join(): the
// main stream waits for them.  A scope left in between (an error of a launch) waits on
// the host for the side streams, whose kernels use buffers that the caller gives back.
class SideFork {
 public:
  SideFork(cudaStream_t main, cudaEvent_t fork_ev, const cudaStream_t* side, const cudaEvent_t* join_ev, int n)
      : main_(main), fork_ev_(fork_ev), side_(side), join_ev_(join_ev), n_(n) {}
  SideFork(const SideFork&) = delete;
  SideFork& operator=(const SideFork&) = delete;
  ~SideFork() {
    if (!open_) return;
    for (int i = 0; i < n_; ++i) (void)cudaStreamSynchronize(side_[i]);
  }
  cudaError_t fork() {
    cudaError_t e = cudaEventRecord(fork_ev_, main_);
    open_ = e == cudaSuccess;
    for (int i = 0; i < n_ && e == cudaSuccess; ++i) e = cudaStreamWaitEvent(side_[i], fork_ev_, 0);
    return e;
  }
  cudaError_t join() {
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < n_ && e == cudaSuccess; ++i) {
      e = cudaEventRecord(join_ev_[i], side_[i]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, join_ev_[i], 0);
    }
    if (e == cudaSuccess) open_ = false;
    return e;
  }

 private:
  cudaStream_t main_;
  cudaEvent_t fork_ev_;
  const cudaStream_t* side_;
  const cudaEvent_t* join_ev_;
  int n_;
  bool open_ = false;
};

}  // namespace gbhf
