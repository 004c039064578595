"""The caching device allocator (devmem.cpp) on the host, compiled against a
stand-in for the driver that has 100 GB and counts: an allocation that does
not fit reclaims what other live threads keep idle, and the idle blocks of all
threads together stay within the process's bound."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "deepaw-half_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "common.h"
#include "devmem.h"

static std::mutex mu;
static std::map<void*, size_t> live;
static size_t used = 0, next_address = 4096;
static size_t capacity = size_t(100) << 30;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> l(mu);
  if (used + n > capacity) return cudaErrorMemoryAllocation;
  *p = reinterpret_cast<void*>(next_address);
  next_address += n;
  used += n;
  live[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> l(mu);
  used -= live.at(p);
  live.erase(p);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "out of memory"; }
}

// n threads that each allocate and free `blocks` blocks of `bytes`, then stay until told to end
struct Sleepers {
  std::mutex m;
  std::condition_variable cv;
  bool end = false;
  int ready = 0;
  std::vector<std::thread> pool;
  Sleepers(int n, int blocks, size_t bytes) {
    for (int t = 0; t < n; ++t)
      pool.emplace_back([=] {
        std::vector<std::pair<void*, size_t>> b(blocks);
        for (auto& x : b) x.first = hb::device_alloc(bytes, &x.second);
        for (auto& x : b) hb::device_free(x.first, x.second);
        std::unique_lock<std::mutex> l(m);
        ++ready;
        cv.notify_all();
        cv.wait(l, [&] { return end; });
      });
    std::unique_lock<std::mutex> l(m);
    cv.wait(l, [&] { return ready == n; });
  }
  ~Sleepers() {
    { std::lock_guard<std::mutex> l(m); end = true; }
    cv.notify_all();
    for (auto& t : pool) t.join();
  }
};

int main() {
  size_t g = 0;
  {
    Sleepers s(3, 6, size_t(5) << 30);   // 30 GB requested and freed by each
    try {
      void* p = hb::device_alloc(size_t(90) << 30, &g);
      hb::device_free(p, g);
    } catch (const hb::Error& e) {
      std::printf("reclaim: %s\n", e.what());
      return 1;
    }
  }
  hb::device_cache_release();
  if (used != 0) { std::printf("release left %zu bytes\n", used); return 2; }
  capacity = size_t(400) << 30;
  {
    Sleepers s(9, 8, size_t(3) << 30);   // 24 GB each, 216 GB in all
    if (used > (size_t(96) << 30)) { std::printf("idle: %zu bytes\n", used); return 3; }
  }
  hb::device_cache_release();
  if (used != 0) { std::printf("release left %zu bytes\n", used); return 4; }
  std::printf("ok\n");
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_cache_is_bounded_and_reclaimed_across_threads(tmp_path):
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or
                                                                        "/usr/local/cuda/bin/nvcc"))), "include")
    src, exe = tmp_path / "cache.cpp", tmp_path / "cache"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, "-I" + cuda, str(src),
                    os.path.join(CSRC, "devmem.cpp"), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
