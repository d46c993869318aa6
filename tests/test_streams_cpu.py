"""Forked launch streams (csrc/streams.h) against a recording stand-in for the CUDA runtime: whatever leaves the
scope, the caller's stream waits for every stream that was forked; calls that overlap hold different sets."""
import os
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gradscf_b200" / "csrc"

RUNTIME = r"""
#pragma once
#include <map>
#include <set>
// A stream's clock counts its operations; an event holds the operations it was recorded after.
typedef int cudaError_t;
const cudaError_t cudaSuccess = 0;
struct FakeStream { std::set<int> done; };
struct FakeEvent { std::set<int> done; };
typedef FakeStream* cudaStream_t;
typedef FakeEvent* cudaEvent_t;
const unsigned cudaStreamNonBlocking = 1, cudaEventDisableTiming = 2;
inline int g_op = 0, g_fail_wait = -1, g_waits = 0, g_live = 0;
inline const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = new FakeStream; ++g_live; return 0; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = new FakeEvent; ++g_live; return 0; }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { delete s; --g_live; return 0; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; --g_live; return 0; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { e->done = s->done; return 0; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (g_waits++ == g_fail_wait) return 1;
  s->done.insert(e->done.begin(), e->done.end());
  return 0;
}
inline int queue_op(cudaStream_t s) { s->done.insert(++g_op); return g_op; }
"""

MAIN = r"""
#include "streams.h"
#include <cstdio>
using namespace b200jk;
static int bad = 0;
#define CHECK(x) do { if (!(x)) { std::printf("failed: %s (line %d)\n", #x, __LINE__); ++bad; } } while (0)

int main() {
  {
    AuxStreams aux;
    aux.create();
    FakeStream st;
    // every stream starts after the caller's work, and the caller continues after all of them
    const int before = queue_op(&st);
    {
      StreamFork f(&aux, &st);
      CHECK(f.count() == kAuxStreams + 1 && f[0] == &st);
      for (int i = 1; i < f.count(); ++i) CHECK(f[i]->done.count(before));
      std::set<int> ops;
      for (int i = 0; i < f.count(); ++i) ops.insert(queue_op(f[i]));
      f.join();
      for (int op : ops) CHECK(st.done.count(op));
    }
    // a launch that throws half way: the same holds for what was queued before it
    std::set<int> ops;
    bool thrown = false;
    try {
      StreamFork f(&aux, &st);
      for (int i = 0; i < f.count(); ++i) ops.insert(queue_op(f[i]));
      throw 7;
    } catch (int) { thrown = true; }
    CHECK(thrown);
    for (int op : ops) CHECK(st.done.count(op));
    // the second of the forks fails: an error, the first one joined
    const int inner = queue_op(aux.s[0]);
    g_waits = 0;
    g_fail_wait = 1;
    thrown = false;
    try { StreamFork f(&aux, &st); } catch (const std::runtime_error&) { thrown = true; }
    CHECK(thrown && st.done.count(inner));
    g_fail_wait = -1;
    // no auxiliary streams: the caller's alone
    StreamFork f(nullptr, &st);
    CHECK(f.count() == 1 && f[0] == &st);
    f.join();
  }
  CHECK(g_live == 0);
  return bad;
}
"""

POOL = r"""
#include "streams.h"
#include <cstdio>
#include <thread>
using namespace b200jk;

int main() {
  int bad = 0;
  {
    StreamPool pool;
    AuxStreams *a, *b;
    {
      StreamPool::Lease x(pool), y(pool);   // two calls at a time
      a = x.get();
      b = y.get();
      if (a == b || a->fork == b->fork || a->s[0] == b->s[0]) ++bad;
    }
    StreamPool::Lease z(pool);              // a later call takes an idle set
    if (z.get() != a && z.get() != b) ++bad;
    // interleaved as two threads may be: B's fork is recorded between A's record and A's waits
    FakeStream sa, sb;
    const int work = queue_op(&sa);
    StreamPool::Lease w(pool);
    cudaEventRecord(z.get()->fork, &sa);
    cudaEventRecord(w.get()->fork, &sb);
    cudaStreamWaitEvent(z.get()->s[0], z.get()->fork, 0);
    if (!z.get()->s[0]->done.count(work)) ++bad;
  }
  if (g_live != 0) ++bad;
  {
    StreamPool pool;                        // idle sets are bounded
    std::vector<std::unique_ptr<StreamPool::Lease>> held;
    for (int i = 0; i < 9; ++i) held.emplace_back(new StreamPool::Lease(pool));
    held.clear();
    if (g_live != 4 * (2 * kAuxStreams + 1)) ++bad;
  }
  if (g_live != 0) ++bad;
  if (bad) std::printf("%d failed\n", bad);
  return bad;
}
"""


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    root = tmp_path_factory.mktemp("streams")
    (root / "cuda_runtime.h").write_text(RUNTIME)
    return root


def run(root, source, name):
    src, exe = root / f"{name}.cc", root / name
    src.write_text(source)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-pthread", "-I", str(root), "-I", str(CSRC),
                    str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout + done.stderr


def test_every_exit_of_a_fork_joins_its_streams(runtime):
    run(runtime, MAIN, "fork")


def test_overlapping_calls_hold_different_streams(runtime):
    run(runtime, POOL, "pool")
