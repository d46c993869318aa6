// Independent launches spread over a caller's stream and auxiliary streams
// that are forked from it and joined back.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

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

// Sets for calls that share nothing else and may overlap from any threads and
// streams: each holds a set of its own (two records of one fork event between
// a record and its waits would drop the order of the first).  Up to kKeep
// idle sets stay for the next call, whose work then queues behind what is
// still running on them.
class StreamPool {
 public:
  class Lease {
   public:
    explicit Lease(StreamPool& pool) : pool_(pool), set_(pool.take()) {}
    ~Lease() { pool_.give_back(std::move(set_)); }
    Lease(const Lease&) = delete;
    Lease& operator=(const Lease&) = delete;
    AuxStreams* get() const { return set_.get(); }

   private:
    StreamPool& pool_;
    std::unique_ptr<AuxStreams> set_;
  };
  StreamPool() { idle_.reserve(kKeep); }

 private:
  static constexpr size_t kKeep = 4;
  std::unique_ptr<AuxStreams> take() {
    std::unique_ptr<AuxStreams> set;
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (!idle_.empty()) {
        set = std::move(idle_.back());
        idle_.pop_back();
        return set;
      }
    }
    set.reset(new AuxStreams());
    set->create();
    return set;
  }
  void give_back(std::unique_ptr<AuxStreams> set) {
    std::lock_guard<std::mutex> lock(mu_);
    if (idle_.size() < kKeep) idle_.push_back(std::move(set));   // else destroyed; its work still completes
  }
  std::mutex mu_;
  std::vector<std::unique_ptr<AuxStreams>> idle_;
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
