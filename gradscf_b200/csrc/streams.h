// Independent launches spread over a caller's stream and auxiliary streams
// that are forked from it and joined back.
#pragma once
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

namespace b200jk {

#ifndef B200JK_AUX_STREAMS
#define B200JK_AUX_STREAMS 3
#endif
constexpr int kAuxStreams = B200JK_AUX_STREAMS;  // streams besides the caller's for concurrent class-pair launches

inline void stream_ok(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// One set of auxiliary streams with the events of its forks and joins.
struct AuxStreams {
  cudaStream_t s[kAuxStreams] = {};
  cudaEvent_t fork = nullptr, join[kAuxStreams] = {};
  AuxStreams() = default;
  AuxStreams(const AuxStreams&) = delete;
  AuxStreams& operator=(const AuxStreams&) = delete;
  void create() {
    for (int i = 0; i < kAuxStreams; ++i) {
      stream_ok(cudaStreamCreateWithFlags(&s[i], cudaStreamNonBlocking), "cudaStreamCreate");
      stream_ok(cudaEventCreateWithFlags(&join[i], cudaEventDisableTiming), "cudaEventCreate");
    }
    stream_ok(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming), "cudaEventCreate");
  }
  ~AuxStreams() {
    for (int i = 0; i < kAuxStreams; ++i) {
      if (s[i]) cudaStreamDestroy(s[i]);
      if (join[i]) cudaEventDestroy(join[i]);
    }
    if (fork) cudaEventDestroy(fork);
  }
};

// The streams of `aux` forked from `st` for the life of this object.  join()
// makes `st` wait for them; a scope that is left by an exception joins too,
// so work already queued on them stays ordered before whatever the caller
// does next on `st` (its buffers may be freed there, a capture may end).
// Without `aux` everything stays on `st`.
class StreamFork {
 public:
  StreamFork(AuxStreams* aux, cudaStream_t st) : aux_(aux), st_(st) {
    if (!aux_) return;
    stream_ok(cudaEventRecord(aux_->fork, st_), "fork");
    for (forked_ = 0; forked_ < kAuxStreams; ++forked_) {
      const cudaError_t e = cudaStreamWaitEvent(aux_->s[forked_], aux_->fork, 0);
      if (e != cudaSuccess) {
        rejoin();
        stream_ok(e, "fork");
      }
    }
  }
  ~StreamFork() { rejoin(); }
  StreamFork(const StreamFork&) = delete;
  StreamFork& operator=(const StreamFork&) = delete;
  int count() const { return aux_ ? kAuxStreams + 1 : 1; }
  cudaStream_t operator[](int i) const { return i == 0 ? st_ : aux_->s[i - 1]; }
  void join() { stream_ok(rejoin(), "join"); }

 private:
  cudaError_t rejoin() {
    cudaError_t first = cudaSuccess;
    for (int i = 0; i < forked_; ++i) {
      cudaError_t e = cudaEventRecord(aux_->join[i], aux_->s[i]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st_, aux_->join[i], 0);
      if (first == cudaSuccess) first = e;
    }
    forked_ = 0;
    return first;
  }
  AuxStreams* aux_;
  cudaStream_t st_;
  int forked_ = 0;
};

}  // namespace b200jk
