// Caching device allocator (see devmem.h).
#include "devmem.h"

#include <atomic>

#include <cuda_runtime.h>

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <utility>

#include "common.h"

namespace hb {

namespace {

using Key = std::pair<int, size_t>;   // (device, bytes)
using Pool = std::multimap<Key, void*>;

// Cached bytes kept by one thread (a 216-atom mixed solve takes 20 GB in all)
// and by the process: what a batch of four such solves comes back for.  At 80
// GB a batch freed and allocated 20 to 40 blocks a step and took 550 to 583 ms
// per k point, at 96 GB 543 to 550.
constexpr size_t kThreadCap = size_t(32) << 30;
constexpr size_t kProcessCap = size_t(96) << 30;

size_t round_bytes(size_t b) {
  if (b <= (size_t(1) << 20)) return (b + 511) & ~size_t(511);
  return (b + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);
}

void timed_free(void* p, size_t bytes) {
  AllocTimer timer("cudaFree", bytes);
  cudaFree(p);
}

struct ThreadCache;

std::mutex g_mu;                       // guards g_pool and g_caches; taken before a cache's own mutex
Pool g_pool;
std::set<ThreadCache*> g_caches;       // of the live threads
std::atomic<size_t> g_cached{0};       // bytes in all caches and the pool

// Smallest block in [key.bytes, 2 key.bytes] on the same device, removed from pool.
void* take(Pool& pool, const Key& key, size_t* granted) {
  auto it = pool.lower_bound(key);
  if (it == pool.end() || it->first.first != key.first || it->first.second > 2 * key.second) return nullptr;
  void* p = it->second;
  *granted = it->first.second;
  pool.erase(it);
  return p;
}

struct ThreadCache {
  std::mutex mu;   // another thread takes it only to give everything back
  Pool pool;
  size_t bytes = 0;
  ThreadCache() {
    std::lock_guard<std::mutex> lock(g_mu);
    g_caches.insert(this);
  }
  ~ThreadCache() {
    if (!pool.empty()) cudaDeviceSynchronize();   // every use of these blocks has finished
    std::lock_guard<std::mutex> lock(g_mu);
    g_caches.erase(this);
    std::lock_guard<std::mutex> own(mu);
    for (auto& kv : pool) g_pool.insert(kv);
    pool.clear();
  }
};

thread_local ThreadCache t_cache;
std::atomic<long long> g_requests{0}, g_driver_allocs{0}, g_refused{0};
std::atomic<size_t> g_refuse_above{0};

void release_all_locked(Pool& pool) {
  for (auto& kv : pool) {
    timed_free(kv.second, kv.first.second);
    g_cached.fetch_sub(kv.first.second);
  }
  pool.clear();
}

}  // namespace

void* device_try_alloc(size_t bytes, size_t* granted) {
  g_requests.fetch_add(1, std::memory_order_relaxed);
  if (const size_t most = g_refuse_above.load(std::memory_order_relaxed); most != 0 && bytes > most) {
    g_refused.fetch_add(1);
    return nullptr;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  const Key key{dev, round_bytes(bytes)};
  {
    std::lock_guard<std::mutex> own(t_cache.mu);
    if (void* p = take(t_cache.pool, key, granted)) {
      t_cache.bytes -= *granted;
      g_cached.fetch_sub(*granted);
      return p;
    }
  }
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (void* p = take(g_pool, key, granted)) {
      g_cached.fetch_sub(*granted);
      return p;
    }
  }
  void* p = nullptr;
  cudaError_t e;
  {
    AllocTimer timer("cudaMalloc", key.second);
    g_driver_allocs.fetch_add(1, std::memory_order_relaxed);
    e = cudaMalloc(&p, key.second);
  }
  if (e != cudaSuccess) {   // give the cache back and retry once
    cudaGetLastError();
    device_cache_release();
    AllocTimer timer("cudaMalloc", key.second);
    g_driver_allocs.fetch_add(1, std::memory_order_relaxed);
    e = cudaMalloc(&p, key.second);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  *granted = key.second;
  return p;
}

void* device_alloc(size_t bytes, size_t* granted) {
  void* p = device_try_alloc(bytes, granted);
  if (!p) fail(kInternal, "device allocation of " + std::to_string(bytes) + " bytes failed: out of memory");
  return p;
}

void device_free(void* p, size_t granted) {
  if (!p) return;
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> own(t_cache.mu);
    if (t_cache.bytes + granted <= kThreadCap) {
      if (g_cached.fetch_add(granted) + granted <= kProcessCap) {
        t_cache.pool.insert({Key{dev, granted}, p});
        t_cache.bytes += granted;
        return;
      }
      g_cached.fetch_sub(granted);
    }
  }
  timed_free(p, granted);
}

long long device_refuse_above(size_t bytes) {
  g_refuse_above.store(bytes);
  return g_refused.exchange(0);
}

void device_alloc_counts(long long* requests, long long* driver_allocations) {
  if (requests) *requests = g_requests.load(std::memory_order_relaxed);
  if (driver_allocations) *driver_allocations = g_driver_allocs.load(std::memory_order_relaxed);
}

// Another thread's cached blocks may still be used by work on its stream:
// cudaFree waits for that.
void device_cache_release() {
  cudaDeviceSynchronize();
  std::lock_guard<std::mutex> lock(g_mu);
  for (ThreadCache* c : g_caches) {
    std::lock_guard<std::mutex> own(c->mu);
    release_all_locked(c->pool);
    c->bytes = 0;
  }
  release_all_locked(g_pool);
}

}  // namespace hb
