// Stand-in for the CUDA runtime in host tests: streams and events are numbers, and
// every call is written to fake_log; call number fake_fail_at (from 1) returns an error.
#pragma once
#include <string>
#include <vector>
using cudaStream_t = int;
using cudaEvent_t = int;
enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 999 };
inline std::vector<std::string> fake_log;
inline int fake_fail_at = 0;
inline cudaError_t fake_call(const std::string& what) {
  fake_log.push_back(what);
  return (int)fake_log.size() == fake_fail_at ? cudaErrorUnknown : cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return fake_call("record " + std::to_string(e) + " on " + std::to_string(s));
}
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  return fake_call("wait " + std::to_string(s) + " for " + std::to_string(e));
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { return fake_call("sync " + std::to_string(s)); }
