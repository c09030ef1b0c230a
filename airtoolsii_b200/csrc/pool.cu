// Device and page-locked memory kept between uses.
//
// cudaMalloc and cudaFree map and unmap pages: making the operator of
// paralleltomo N = 512, 180 angles x 724 rays, projecting and back-projecting
// with it took 18-24 ms, 4.9 ms of it kernels, and the first solve on a new
// operator 2-4 ms more than the second.  Blocks given up are therefore kept
// and handed out again for requests of about their size (sizes are rounded up
// to sixteenths of a power of two, so that problems whose nonzeros differ a
// little share blocks).
//
// The kept blocks are bounded (kKeepBytes per device), those that nobody
// asked for during the last kKeepCalls calls go back to the device, and all
// of them do when an allocation fails.  Giving a block up waits for the
// device as cudaFree does, so a kept block has no work in flight on any
// stream; the lists are guarded by a mutex.
#include <map>
#include <mutex>
#include <unordered_map>

#include "common.cuh"

namespace airt {

namespace {

constexpr size_t kKeepBytes = (size_t)6 << 30;
constexpr uint64_t kKeepCalls = 512;
constexpr size_t kKeepPinned = 64;

struct Block {
  void *p;
  uint64_t when;  // call count at which it was given up
};

struct Pool {
  std::mutex mu;
  // per device: kept blocks by size, and their total
  std::map<int, std::multimap<size_t, Block>> kept;
  std::map<int, size_t> bytes;
  std::unordered_map<void *, std::pair<size_t, int>> used;  // size and device of handed-out blocks
  std::vector<void *> pinned;
  uint64_t calls = 0;
};

Pool &pool() {
  static Pool *p = new Pool();  // outlives every static that might free memory
  return *p;
}

size_t rounded(size_t n) {
  if (n <= 512) return 512;
  size_t top = 512;
  while (top * 2 <= n) top *= 2;
  const size_t step = top / 16 < 512 ? 512 : top / 16;
  return (n + step - 1) / step * step;
}

// Gives kept blocks of `dev` back: all of them, or those unused for long.
void trim(Pool &P, int dev, bool all) {
  auto &m = P.kept[dev];
  for (auto it = m.begin(); it != m.end();) {
    if (all || P.calls - it->second.when > kKeepCalls) {
      cudaFree(it->second.p);
      P.bytes[dev] -= it->first;
      it = m.erase(it);
    } else {
      ++it;
    }
  }
}

}  // namespace

void *device_alloc(size_t bytes, cudaError_t *err) {
  Pool &P = pool();
  int dev = 0;
  *err = cudaGetDevice(&dev);
  if (*err != cudaSuccess) return nullptr;
  const size_t n = rounded(bytes);
  std::lock_guard<std::mutex> lock(P.mu);
  ++P.calls;
  auto &m = P.kept[dev];
  auto it = m.lower_bound(n);
  void *p = nullptr;
  size_t size = n;
  if (it != m.end() && it->first <= n + n / 8) {
    p = it->second.p;
    size = it->first;
    P.bytes[dev] -= size;
    m.erase(it);
  } else {
    *err = cudaMalloc(&p, n);
    if (*err == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      trim(P, dev, true);
      *err = cudaMalloc(&p, n);
    }
    if (*err != cudaSuccess) return nullptr;
  }
  P.used[p] = {size, dev};
  return p;
}

void device_free(void *p) {
  if (!p) return;
  cudaDeviceSynchronize();
  Pool &P = pool();
  std::lock_guard<std::mutex> lock(P.mu);
  ++P.calls;
  auto it = P.used.find(p);
  if (it == P.used.end()) return;
  const size_t size = it->second.first;
  const int dev = it->second.second;
  P.used.erase(it);
  int cur = 0;
  cudaGetDevice(&cur);
  // a block of another device is not idle after the wait above
  if (cur != dev || P.bytes[dev] + size > kKeepBytes) {
    cudaFree(p);
  } else {
    P.kept[dev].insert({size, Block{p, P.calls}});
    P.bytes[dev] += size;
  }
  if (P.calls % 64 == 0) trim(P, cur, false);
}

void *pinned_alloc(cudaError_t *err) {
  Pool &P = pool();
  std::lock_guard<std::mutex> lock(P.mu);
  *err = cudaSuccess;
  if (!P.pinned.empty()) {
    void *p = P.pinned.back();
    P.pinned.pop_back();
    return p;
  }
  void *p = nullptr;
  *err = cudaMallocHost(&p, kPinnedBytes);
  return *err == cudaSuccess ? p : nullptr;
}

void pinned_free(void *p) {
  if (!p) return;
  Pool &P = pool();
  std::lock_guard<std::mutex> lock(P.mu);
  if (P.pinned.size() < kKeepPinned) P.pinned.push_back(p);
  else cudaFreeHost(p);
}

}  // namespace airt
