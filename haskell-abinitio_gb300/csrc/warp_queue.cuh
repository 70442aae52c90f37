// The queue of surviving kets that a warp keeps in shared memory (screen.cuh): at most
// 31 are left when a group of 32 is scanned, so 64 slots hold it.  The slots a batch
// takes are [0, nk), nk = min(queued, 32), and the rest moves down.
#pragma once

namespace gbhf {

constexpr int QUEUE_SLOTS = 64;

// Append the lanes' kets that pass to the warp's queue (at most 31 queued before).
__device__ __forceinline__ void queue_push(int* q, int& queued, int jk, bool pass, int lane) {
  const unsigned m = __ballot_sync(0xffffffffu, pass);
  if (pass) q[queued + __popc(m & ((1u << lane) - 1))] = jk;
  queued += __popc(m);
  __syncwarp();
}
// Remove the first nk (at most 31 are left).
__device__ __forceinline__ void queue_pop(int* q, int& queued, int nk, int lane) {
  queued -= nk;
  __syncwarp();
  const int v = lane < queued ? q[nk + lane] : 0;
  __syncwarp();
  if (lane < queued) q[lane] = v;
  __syncwarp();
}
// The ket that a lane of the batch takes, kets on the low lg bits of the lane; lanes
// beyond the batch point at the task's first ket and keep none.  Every ket comes from
// the scan of [first, first + count).  One that does not is dropped and reported (bad):
// the (dd|ss) instance of this form, not in use, read out of bounds on the device, and
// neither reading nor the host test of this queue showed why.
__device__ __forceinline__ int queue_ket(const int* q, int nk, int lg, int lane, int first, int count, bool& keep,
                                         bool& bad) {
  const int slot = lane & ((1 << lg) - 1);
  keep = slot < nk;
  const int jk = keep ? q[slot] : first;
  bad = (unsigned)(jk - first) >= (unsigned)count;
  keep = keep && !bad;
  return bad ? first : jk;
}

}  // namespace gbhf
