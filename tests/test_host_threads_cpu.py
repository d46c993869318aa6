"""Host work on several threads (csrc/host_threads.h): every index runs once, an exception comes back to the caller,
and memory or threads that run out while the threads are being started end neither the process nor the work."""
import os
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "gradscf_b200" / "csrc"

MAIN = r"""
#include "host_threads.h"
#include <cstdio>
#include <cstdlib>
#include <new>
#include <stdexcept>
// allocations of this thread fail once `left` of them are used up
static thread_local long left = -1;
void* operator new(std::size_t n) {
  if (left >= 0 && left-- == 0) { left = -1; throw std::bad_alloc(); }
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main() {
  int bad = 0;
  for (long fail = -1; fail < 12; ++fail)      // -1: none; 0: the pool itself; then the threads
    for (std::size_t threads : {1, 2, 8})
      for (std::size_t n : {0, 1, 5, 100}) {
        std::vector<std::atomic<int>> ran(n);
        left = fail;
        b200jk::run_indexed(n, threads, [&](std::size_t i) { ++ran[i]; });
        left = -1;
        for (auto& r : ran) bad += r != 1;
      }
  int caught = 0;
  try {
    b200jk::run_indexed(50, 4, [&](std::size_t i) { if (i == 17) throw std::runtime_error("seventeen"); });
  } catch (const std::runtime_error&) { ++caught; }
  if (caught != 1) ++bad;
  if (bad) std::printf("%d failed\n", bad);
  return bad;
}
"""


def test_threads_that_cannot_start_are_done_without(tmp_path):
    src, exe = tmp_path / "threads.cc", tmp_path / "threads"
    src.write_text(MAIN)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, (done.returncode, done.stdout, done.stderr)
