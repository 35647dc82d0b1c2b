"""Copies through pinned slots on the CPU: the header with the copying threads, compiled against a fake of
the CUDA runtime.  The fake's DMAs run in order on a thread of its own, a call from any thread but the one
that started the copy is an error (a stream handle may name another stream there), and a call can be made
to fail."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "poissonreconstruction_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <thread>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999, cudaErrorNotReady = 600 };
enum { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2, cudaEventDisableTiming = 2 };
typedef int cudaStream_t;
struct Event { long at = 0; };
typedef Event* cudaEvent_t;
struct Gpu {
  std::mutex m;
  std::condition_variable cv;
  std::deque<std::function<void()>> q;
  long pushed = 0, done = 0;
  bool quit = false;
  std::thread t{[this] {
    std::unique_lock<std::mutex> l(m);
    for (;;) {
      cv.wait(l, [&] { return quit || !q.empty(); });
      if (q.empty()) return;
      auto f = q.front();
      q.pop_front();
      l.unlock();
      f();
      l.lock();
      ++done;
      cv.notify_all();
    }
  }};
  ~Gpu() {
    { std::lock_guard<std::mutex> l(m); quit = true; }
    cv.notify_all();
    t.join();
  }
};
inline Gpu& gpu() { static Gpu g; return g; }
inline std::thread::id& owner() { static std::thread::id i; return i; }
inline int& fail_in() { static int n = -1; return n; }  // calls until one fails; -1: none does
inline bool fails() {
  if (std::this_thread::get_id() != owner()) { std::puts("a CUDA call from another thread"); std::_Exit(2); }
  return fail_in() >= 0 && fail_in()-- == 0;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaMallocHost(void** p, size_t n) {
  if (fails()) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) {
  if (fails()) return cudaErrorUnknown;
  *e = new Event;
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t) {
  if (fails()) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(gpu().m);
  gpu().q.push_back([=] { std::memcpy(d, s, n); });
  ++gpu().pushed;
  gpu().cv.notify_all();
  return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  if (fails()) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(gpu().m);
  e->at = gpu().pushed;
  return cudaSuccess;
}
inline cudaError_t cudaEventQuery(cudaEvent_t e) {
  if (fails()) return cudaErrorUnknown;
  std::lock_guard<std::mutex> l(gpu().m);
  return gpu().done >= e->at ? cudaSuccess : cudaErrorNotReady;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (fails()) return cudaErrorUnknown;
  std::unique_lock<std::mutex> l(gpu().m);
  gpu().cv.wait(l, [&] { return gpu().done >= e->at; });
  return cudaSuccess;
}
inline void drain() {
  std::unique_lock<std::mutex> l(gpu().m);
  gpu().cv.wait(l, [&] { return gpu().done >= gpu().pushed; });
}
"""

MAIN = r"""
#include "pr_staged_copy.h"

typedef std::vector<unsigned char> Bytes;

int main() {
  owner() = std::this_thread::get_id();
  for (int k = 0; k <= pr::kStageSlots; ++k) {  // no pinned memory, or no event
    pr::StageSlots st;
    fail_in() = k;
    if (st.make()) return 3;
    fail_in() = -1;
    if (!st.make()) return 4;  // there is some later
    st.free();
  }
  pr::StageSlots st;
  if (!st.make()) return 5;
  const size_t S = pr::kStageSlot;
  int seed = 0, errors = 0;
  for (size_t bytes : {size_t(1), S - 1, S, S + 1, 7 * S, 8 * S, 8 * S + 5, 9 * S, 21 * S + 3})
    for (int nt = 1; nt <= pr::kStageThreads; ++nt)
      for (int fail : {-1, 0, 1, 5, 40}) {
        Bytes a(bytes), dev(bytes), back(bytes);
        unsigned v = (unsigned)++seed * 2654435761u;
        for (auto& x : a) x = (unsigned char)((v = v * 1664525u + 1013904223u) >> 24);
        Bytes src = a;
        fail_in() = fail;
        cudaError_t e = pr::staged_copy(0, st, dev.data(), src.data(), bytes, nt, false);
        std::memset(src.data(), 0, bytes);  // the source is the caller's again
        // the other way at once, through slots whose last DMAs may still run
        if (e == cudaSuccess) e = pr::staged_copy(0, st, dev.data(), back.data(), bytes, nt % 3 + 1, true);
        const bool failed = fail >= 0 && fail_in() < 0;
        fail_in() = -1;
        drain();
        if (failed != (e != cudaSuccess)) return 6;
        if (!failed && (dev != a || back != a)) return 7;
        errors += failed;
      }
  st.free();
  return errors > 0 ? 0 : 8;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_staged_copy_against_a_fake_runtime(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"),
                    "-o", str(exe), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout)


LENT = r"""
#include "pr_staged_copy.h"

int main() {  // slots in the owner's memory, of another size: the owner's bytes around them stay
  owner() = std::this_thread::get_id();
  for (size_t S : {size_t(1) << 12, size_t(192) << 10}) for (size_t n : {1, 4, 8}) {
    std::vector<unsigned char> block((n + 2) * S, 0xa5);
    pr::StageSlots st;
    fail_in() = 0;
    if (st.lend(block.data() + S, S, n)) return 3;  // no event
    fail_in() = -1;
    if (!st.lend(block.data() + S, S, n)) return 4;
    for (size_t bytes : {size_t(1), S - 1, S, S + 1, 8 * S, 8 * S + 5, 21 * S + 3})
      for (int nt = 1; nt <= pr::kStageThreads; ++nt) {
        std::vector<unsigned char> a(bytes), dev(bytes), back(bytes);
        for (size_t i = 0; i < bytes; ++i) a[i] = (unsigned char)(i * 31 + i / S + nt);
        if (pr::staged_copy(0, st, dev.data(), a.data(), bytes, nt, false) != cudaSuccess) return 5;
        if (pr::staged_copy(0, st, dev.data(), back.data(), bytes, nt % 3 + 1, true) != cudaSuccess) return 6;
        drain();
        if (dev != a || back != a) return 7;
      }
    for (size_t i = 0; i < S; ++i)
      if (block[i] != 0xa5 || block[(n + 1) * S + i] != 0xa5) return 8;
    st.free();  // leaves the memory
    block[S] = 1;
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_staged_copy_in_lent_memory(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(LENT)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"),
                    "-o", str(exe), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout)


@pytest.mark.gpu
def test_first_large_copy_of_a_context_costs_no_allocation():
    """A program may make a context for one solve.  Its first copy out does not allocate pinned memory that
    only later ones would pay for (6 ms, where the copy of 2 MB takes 0.3)."""
    import time

    import numpy as np

    import poissonreconstruction_b200 as prb
    from poissonreconstruction_b200 import synthetic
    pts = synthetic.torus(3000, seed=3)
    params = prb.ReconstructParams(depth=6, point_weight=4.0)
    first, later = [], []
    for _ in range(6):
        with prb.Context(0) as c:
            c.solve(pts, params)
            for times in (first, later):
                t = time.perf_counter()
                x = c.coefficients()
                times.append(time.perf_counter() - t)
            assert x.shape == (8 ** 6,) and np.isfinite(x).all()
    assert min(first) < min(later) + 2e-3, (first, later)
