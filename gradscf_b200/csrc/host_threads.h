// Independent host work shared by a few threads.
#pragma once
#include <atomic>
#include <cstddef>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace b200jk {

// f(0) .. f(n - 1), once each, on the calling thread and up to threads - 1
// more; the first exception of an f is rethrown here once all have ended.
// Threads that cannot be started (no threads or no memory for them) are done
// without: what leaves this function never unwinds over a running thread.
template <typename F>
void run_indexed(size_t n, size_t threads, F&& f) {
  std::atomic<size_t> next{0};
  std::mutex mu;
  std::exception_ptr failed;
  auto run = [&] {
    try {
      for (size_t i; (i = next++) < n;) f(i);
    } catch (...) {
      std::lock_guard<std::mutex> lock(mu);
      if (!failed) failed = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  try {
    pool.reserve(threads);
    while (pool.size() + 1 < threads) pool.emplace_back(run);
  } catch (...) {
  }
  run();
  for (auto& t : pool) t.join();
  if (failed) std::rethrow_exception(failed);
}

}  // namespace b200jk
