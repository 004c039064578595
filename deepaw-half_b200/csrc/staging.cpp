// Staged copies of band blocks (see staging.h).
//
// A copy from or to pageable memory goes through the driver's own staging on
// the calling thread: 11-12 GB/s on the B200 hosts, and for a fresh output
// array that thread also takes every page fault.  Here a few host threads
// move pieces between the caller's memory and pinned buffers, each issuing
// its own device copy, so the host copies (and faults) run in parallel and
// overlap the PCIe transfers: 160 bands of the 64-atom cell, 28 MB in and
// 2 x 28 MB out, 16.3 -> 9.5 ms for the whole half_apply_hs call (with the
// faster basis build and without an explicit fill of the outputs).
//
// The pinned buffers belong to the process: at most kMaxSlots of kPiece
// bytes, taken by one copy at a time, and freed with the last context.  A
// copy that finds none free, or that is too small to gain, takes the
// driver's path; so does memory that is already pinned, and anything else
// that is not ordinary host memory.
#include "staging.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace hb {

namespace {

constexpr size_t kPiece = size_t(2) << 20;      // bytes of a pinned buffer
constexpr size_t kMinPiece = size_t(256) << 10; // smallest piece worth a thread
constexpr size_t kMinBytes = size_t(8) << 20;    // below this the driver's path is faster (2 MB blocks: 165 against 310 us)
constexpr int kThreads = 8;                     // pieces in flight per copy
constexpr int kMaxSlots = 4 * kThreads;         // 64 MB of pinned memory: four copies at once

struct Slot {
  void* p = nullptr;
  cudaEvent_t done = nullptr;   // the last device copy that reads or writes p
  int device = 0;
};

std::mutex g_mu;
std::vector<Slot> g_free;
int g_slots = 0;

// Up to `want` buffers for the current device; fewer, or none, when others hold them.
std::vector<Slot> take_slots(int want) {
  std::vector<Slot> got;
  int dev = 0;
  HALF_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(g_mu);
  for (size_t i = g_free.size(); i-- > 0 && int(got.size()) < want;)
    if (g_free[i].device == dev) {
      got.push_back(g_free[i]);
      g_free.erase(g_free.begin() + long(i));
    }
  while (int(got.size()) < want && g_slots < kMaxSlots) {
    Slot s;
    s.device = dev;
    if (cudaHostAlloc(&s.p, kPiece, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      break;
    }
    if (cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming) != cudaSuccess) {
      cudaGetLastError();
      cudaFreeHost(s.p);
      break;
    }
    ++g_slots;
    got.push_back(s);
  }
  return got;
}

void give_slots(const std::vector<Slot>& slots) {
  std::lock_guard<std::mutex> lock(g_mu);
  g_free.insert(g_free.end(), slots.begin(), slots.end());
}

bool ordinary_host_memory(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// Runs move(first column, columns, slot) over all pieces on up to kThreads
// threads, this one among them; false when the copy should take the driver's path.
template <typename Move>
bool in_pieces(const void* host, long long n, long long cols, Move move) {
  const size_t col = size_t(n) * sizeof(double2);
  if (col == 0 || cols <= 0 || col > kPiece || col * size_t(cols) < kMinBytes || !ordinary_host_memory(host)) return false;
  const int cores = std::max(1, int(std::thread::hardware_concurrency()) / 2);
  const long long most = (long long)std::max<size_t>(1, kPiece / col);
  const long long least = (long long)((kMinPiece + col - 1) / col);
  const long long per = std::min(most, std::max(least, (cols + kThreads - 1) / kThreads));
  const long long pieces = (cols + per - 1) / per;
  std::vector<Slot> slots = take_slots(int(std::min<long long>(std::min(kThreads, cores), pieces)));
  if (slots.empty()) return false;
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<long long> next{0};
  std::atomic<int> failed{int(cudaSuccess)};
  auto work = [&](const Slot& slot) {
    cudaError_t e = cudaSetDevice(dev);
    while (e == cudaSuccess && failed.load() == int(cudaSuccess)) {
      const long long i = next.fetch_add(1);
      if (i >= pieces) break;
      e = move(i * per, std::min(per, cols - i * per), slot);
    }
    if (e != cudaSuccess) failed.store(int(e));
  };
  std::vector<std::thread> pool;
  try {
    for (size_t t = 1; t < slots.size(); ++t) pool.emplace_back(work, slots[t]);
  } catch (...) {   // no more threads: the ones that run, and this one, do the rest
  }
  work(slots[0]);
  for (auto& t : pool) t.join();
  for (auto& s : slots)   // also on failure: nothing may still use a buffer that is given back
    if (failed.load() != int(cudaSuccess)) cudaEventSynchronize(s.done);
  give_slots(slots);
  cuda_check(cudaError_t(failed.load()), "staged copy");
  return true;
}

}  // namespace

void block_to_device(double2* dst, const void* src, long long ld, long long n, long long cols, cudaStream_t s) {
  const size_t col = size_t(n) * sizeof(double2), pitch = size_t(ld) * sizeof(double2);
  const char* from = static_cast<const char*>(src);
  const bool staged = in_pieces(src, n, cols, [&](long long c0, long long nc, const Slot& slot) {
    cudaError_t e = cudaEventSynchronize(slot.done);   // the buffer's last copy has left it
    if (e != cudaSuccess) return e;
    if (ld == n) {
      std::memcpy(slot.p, from + size_t(c0) * pitch, size_t(nc) * col);
    } else {
      for (long long c = 0; c < nc; ++c)
        std::memcpy(static_cast<char*>(slot.p) + size_t(c) * col, from + size_t(c0 + c) * pitch, col);
    }
    e = cudaMemcpyAsync(dst + c0 * n, slot.p, size_t(nc) * col, cudaMemcpyHostToDevice, s);
    return e == cudaSuccess ? cudaEventRecord(slot.done, s) : e;
  });
  if (!staged)
    HALF_CUDA(cudaMemcpy2DAsync(dst, col, src, pitch, col, size_t(cols), cudaMemcpyHostToDevice, s));
}

void block_to_host(void* dst, long long ld, const double2* src, long long n, long long cols, cudaStream_t s) {
  const size_t col = size_t(n) * sizeof(double2), pitch = size_t(ld) * sizeof(double2);
  char* to = static_cast<char*>(dst);
  const bool staged = in_pieces(dst, n, cols, [&](long long c0, long long nc, const Slot& slot) {
    cudaError_t e = cudaEventSynchronize(slot.done);
    if (e == cudaSuccess) e = cudaMemcpyAsync(slot.p, src + c0 * n, size_t(nc) * col, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaEventRecord(slot.done, s);
    if (e == cudaSuccess) e = cudaEventSynchronize(slot.done);
    if (e != cudaSuccess) return e;
    if (ld == n) {
      std::memcpy(to + size_t(c0) * pitch, slot.p, size_t(nc) * col);
    } else {
      for (long long c = 0; c < nc; ++c)
        std::memcpy(to + size_t(c0 + c) * pitch, static_cast<char*>(slot.p) + size_t(c) * col, col);
    }
    return cudaSuccess;
  });
  if (!staged) {
    HALF_CUDA(cudaMemcpy2DAsync(dst, pitch, src, col, col, size_t(cols), cudaMemcpyDeviceToHost, s));
    HALF_CUDA(cudaStreamSynchronize(s));
  }
}

void staging_release() {
  std::lock_guard<std::mutex> lock(g_mu);
  for (auto& s : g_free) {
    cudaEventSynchronize(s.done);
    cudaEventDestroy(s.done);
    cudaFreeHost(s.p);
    --g_slots;
  }
  g_free.clear();
}

}  // namespace hb
