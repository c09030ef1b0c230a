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
// A block belongs to the CUDA context that it was allocated in and carries
// that context's id (the driver never reuses one): blocks are kept per
// context, and cudaDeviceReset or a context of the caller's own starts with
// none.  A block that is given up while another context is current is freed
// if its context still owns the address, and forgotten if that context is
// gone: the address may be somebody else's by then.
//
// Giving a block up waits for the device as cudaFree does, so a kept block has
// no work in flight on any stream; where that wait fails (a stream of this
// thread is capturing) the block is not kept.  The lists are guarded by a
// mutex.  Kept blocks take at most kKeepBytes and a quarter of the memory that
// is free beside them (asked once a second): the ones given up first make room
// for new ones.  Those that nobody asked for during kKeepSeconds go back to
// the device at the next call, all of them do when an allocation fails and in
// airt_release_memory.
#include <cuda.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <map>
#include <mutex>

#include "../../include/airt.h"
#include "common.cuh"

namespace airt {

namespace {

constexpr size_t kKeepBytes = (size_t)6 << 30, kKeepPinned = 64 * kPinnedBytes;
constexpr size_t kSmallBytes = (size_t)256 << 20;  // kept without asking how much is free
constexpr double kKeepSeconds = 30.0;

// What the pool's bookkeeping needs of the driver.
struct Backend {
  virtual ~Backend() = default;
  virtual unsigned long long context() = 0;  // id of the current context; 0: none
  virtual cudaError_t get(size_t bytes, void **p) = 0;
  virtual void put(void *p) = 0;
  virtual bool owns(unsigned long long ctx, void *p) = 0;  // p is memory of the living context ctx
  virtual bool idle() = 0;                                 // no work in flight in the current context
  virtual size_t room() = 0;                               // free memory
  virtual double now() = 0;                                // seconds
};

size_t rounded(size_t n) {
  if (n <= 512) return 512;
  size_t top = 512;
  while (top * 2 <= n) top *= 2;
  const size_t step = top / 16 < 512 ? 512 : top / 16;
  return (n + step - 1) / step * step;
}

class BlockPool {
 public:
  BlockPool(Backend &backend, size_t keep) : be(backend), keep_bytes(keep) {}

  DevBlock alloc(size_t bytes, cudaError_t *err) {
    DevBlock b{nullptr, rounded(bytes), be.context()};
    std::lock_guard<std::mutex> lock(mu);
    trim(b.ctx, false);
    Kept &k = kept[b.ctx];
    auto it = b.ctx ? k.blocks.lower_bound(b.size) : k.blocks.end();
    if (it != k.blocks.end() && it->first <= b.size + b.size / 8) {
      b.p = it->second.p;
      b.size = it->first;
      k.bytes -= b.size;
      k.blocks.erase(it);
      *err = cudaSuccess;
      return b;
    }
    *err = be.get(b.size, &b.p);
    if (*err == cudaErrorMemoryAllocation) {
      trim(b.ctx, true);
      *err = be.get(b.size, &b.p);
    }
    if (*err != cudaSuccess) b.p = nullptr;
    else if (!b.ctx) b.ctx = be.context();
    return b;
  }

  void give(const DevBlock &b) noexcept {
    if (!b.p) return;
    const unsigned long long cur = be.context();
    if (cur != b.ctx || !cur) {
      if (cur && be.owns(b.ctx, b.p)) be.put(b.p);
      return;
    }
    const bool idle = be.idle();
    std::lock_guard<std::mutex> lock(mu);
    try {
      trim(cur, false);
      Kept &k = kept[cur];
      const size_t total = k.bytes + b.size;
      const double t = be.now();
      // asking for every block took the session above from 6.1 to 8-11 ms
      if (total > kSmallBytes && t - k.asked >= 1.0) {
        k.limit = std::min(keep_bytes, be.room() / 4);
        k.asked = t;
      }
      const size_t limit = std::min(keep_bytes, std::max(k.limit, kSmallBytes));
      if (idle && b.size <= limit) {
        while (k.bytes + b.size > limit) drop_oldest(k);
        k.blocks.insert({b.size, Block{b.p, t}});
        k.bytes += b.size;
        return;
      }
    } catch (...) {  // no host memory for the list
    }
    be.put(b.p);
  }

  // Frees the current context's kept blocks and forgets those of contexts that are gone.
  void release() {
    const unsigned long long cur = be.context();
    std::lock_guard<std::mutex> lock(mu);
    trim(cur, true);
    for (auto c = kept.begin(); c != kept.end();) {
      if (c->first != cur)
        for (auto it = c->second.blocks.begin(); it != c->second.blocks.end();) {
          if (be.owns(c->first, it->second.p)) {
            ++it;
          } else {
            c->second.bytes -= it->first;
            it = c->second.blocks.erase(it);
          }
        }
      c = c->second.blocks.empty() ? kept.erase(c) : std::next(c);
    }
  }

 private:
  struct Block {
    void *p;
    double when;  // when it was given up
  };
  struct Kept {
    std::multimap<size_t, Block> blocks;
    size_t bytes = 0;
    size_t limit = 0;                       // a quarter of the memory that was free ..
    double asked = -INFINITY, looked = 0.0; // .. then; last look at the blocks' age
  };
  Backend &be;
  const size_t keep_bytes;
  std::mutex mu;
  std::map<unsigned long long, Kept> kept;  // by context id

  // Frees the block that was given up first (there is one).
  void drop_oldest(Kept &k) {
    auto old = k.blocks.begin();
    for (auto it = k.blocks.begin(); it != k.blocks.end(); ++it)
      if (it->second.when < old->second.when) old = it;
    be.put(old->second.p);
    k.bytes -= old->first;
    k.blocks.erase(old);
  }

  // Frees kept blocks of the current context `ctx`: all of them, or (looked
  // at once a second) those unused for long.
  void trim(unsigned long long ctx, bool all) {
    auto c = kept.find(ctx);
    if (!ctx || c == kept.end()) return;
    Kept &k = c->second;
    const double t = be.now();
    if (!all && t - k.looked < 1.0) return;
    k.looked = t;
    for (auto it = k.blocks.begin(); it != k.blocks.end();) {
      if (all || t - it->second.when > kKeepSeconds) {
        be.put(it->second.p);
        k.bytes -= it->first;
        it = k.blocks.erase(it);
      } else {
        ++it;
      }
    }
  }
};

// Whether the driver knows p as memory of context ctx.
bool context_owns(unsigned long long ctx, void *p) {
  using Attr = CUresult(CUDAAPI *)(void *, CUpointer_attribute, CUdeviceptr);
  using Id = CUresult(CUDAAPI *)(CUcontext, unsigned long long *);
  void *f = nullptr, *g = nullptr;
  cudaDriverEntryPointQueryResult q, r;
  if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &q) != cudaSuccess || !f ||
      cudaGetDriverEntryPoint("cuCtxGetId", &g, cudaEnableDefault, &r) != cudaSuccess || !g) {
    cudaGetLastError();
    return false;
  }
  CUcontext owner = nullptr;
  if (reinterpret_cast<Attr>(f)(&owner, CU_POINTER_ATTRIBUTE_CONTEXT, (CUdeviceptr)p) != CUDA_SUCCESS || !owner)
    return false;
  unsigned long long id = 0;
  return reinterpret_cast<Id>(g)(owner, &id) == CUDA_SUCCESS && id == ctx;
}

struct DriverBackend : Backend {
  bool pinned;
  explicit DriverBackend(bool page_locked) : pinned(page_locked) {}
  unsigned long long context() override {
    try {
      return current_context_id();
    } catch (...) {  // no device, or the process is shutting down
      return 0;
    }
  }
  cudaError_t get(size_t bytes, void **p) override {
    const cudaError_t e = pinned ? cudaMallocHost(p, bytes) : cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
    return e;
  }
  void put(void *p) override {
    if (pinned) cudaFreeHost(p);
    else cudaFree(p);
  }
  bool owns(unsigned long long ctx, void *p) override { return context_owns(ctx, p); }
  // page-locked blocks: their owner has waited for its stream
  bool idle() override { return pinned || cudaDeviceSynchronize() == cudaSuccess; }
  size_t room() override {
    size_t free = 0, total = 0;
    return cudaMemGetInfo(&free, &total) == cudaSuccess ? free : 0;
  }
  double now() override {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
  }
};

// They outlive every static that might free memory.
BlockPool &device_pool() {
  static BlockPool *p = new BlockPool(*new DriverBackend(false), kKeepBytes);
  return *p;
}
BlockPool &pinned_pool() {
  static BlockPool *p = new BlockPool(*new DriverBackend(true), kKeepPinned);
  return *p;
}

}  // namespace

DevBlock device_alloc(size_t bytes, cudaError_t *err) { return device_pool().alloc(bytes, err); }
void device_free(const DevBlock &b) noexcept { device_pool().give(b); }
DevBlock pinned_alloc(cudaError_t *err) { return pinned_pool().alloc(kPinnedBytes, err); }
void pinned_free(const DevBlock &b) noexcept { pinned_pool().give(b); }

namespace {

// A pool over made-up memory: addresses are numbers, the lowest free one is
// handed out first, and a context's memory goes with it.
struct FakeDevice : Backend {
  std::mutex mu;
  std::map<uintptr_t, std::pair<unsigned long long, size_t>> live;  // address -> context, bytes
  unsigned long long ctx = 1;
  size_t total, used = 0;
  bool quiet = true;
  double clock = 100.0;
  int64_t gets = 0, puts = 0, wrong = 0;
  BlockPool pool{*this, kKeepBytes};
  std::vector<DevBlock> blocks;

  explicit FakeDevice(size_t bytes) : total(bytes) {}
  unsigned long long context() override { return ctx; }
  cudaError_t get(size_t bytes, void **p) override {
    std::lock_guard<std::mutex> lock(mu);
    if (used + bytes > total) return cudaErrorMemoryAllocation;
    uintptr_t at = 4096;
    for (auto &l : live) {
      if (l.first >= at + bytes) break;
      at = l.first + l.second.second;
    }
    live[at] = {ctx, bytes};
    used += bytes;
    ++gets;
    *p = reinterpret_cast<void *>(at);
    return cudaSuccess;
  }
  void put(void *p) override {
    std::lock_guard<std::mutex> lock(mu);
    auto it = live.find(reinterpret_cast<uintptr_t>(p));
    if (it == live.end()) {
      ++wrong;
      return;
    }
    used -= it->second.second;
    live.erase(it);
    ++puts;
  }
  bool owns(unsigned long long c, void *p) override {
    std::lock_guard<std::mutex> lock(mu);
    auto it = live.find(reinterpret_cast<uintptr_t>(p));
    return it != live.end() && it->second.first == c;
  }
  bool idle() override { return quiet; }
  size_t room() override {
    std::lock_guard<std::mutex> lock(mu);
    return total - used;
  }
  double now() override { return clock; }

  int64_t op(int what, int64_t a) {
    switch (what) {
      case 0: ctx = (unsigned long long)a; return 0;
      case 1: quiet = a != 0; return 0;
      case 2: clock += (double)a; return 0;
      case 3: {  // context a is gone
        std::lock_guard<std::mutex> lock(mu);
        for (auto it = live.begin(); it != live.end();) {
          if (it->second.first == (unsigned long long)a) {
            used -= it->second.second;
            it = live.erase(it);
          } else {
            ++it;
          }
        }
        return 0;
      }
      case 4: {
        cudaError_t e;
        const DevBlock b = pool.alloc((size_t)a, &e);
        if (!b.p) return -1;
        std::lock_guard<std::mutex> lock(mu);
        blocks.push_back(b);
        return (int64_t)blocks.size() - 1;
      }
      case 5: {
        DevBlock b;
        {
          std::lock_guard<std::mutex> lock(mu);
          b = blocks.at((size_t)a);
        }
        pool.give(b);
        return 0;
      }
      case 6: pool.release(); return 0;
      case 7: {
        std::lock_guard<std::mutex> lock(mu);
        return (int64_t) reinterpret_cast<uintptr_t>(blocks.at((size_t)a).p);
      }
      case 8: return gets;
      case 9: return puts;
      case 10: return wrong;
      case 11: return (int64_t)used;
    }
    return -2;
  }
};

}  // namespace
}  // namespace airt

using namespace airt;

extern "C" int airt_release_memory(void) {
  try {
    device_pool().release();
    pinned_pool().release();
  } catch (...) {
    set_error("unexpected internal error");
    return AIRT_ERR_CUDA;
  }
  return AIRT_OK;
}

extern "C" void *airt_test_pool_new(int64_t bytes) {
  try {
    return new FakeDevice((size_t)bytes);
  } catch (...) {
    return nullptr;
  }
}

extern "C" int64_t airt_test_pool_op(void *pool, int what, int64_t arg) {
  try {
    return static_cast<FakeDevice *>(pool)->op(what, arg);
  } catch (...) {
    return -3;
  }
}

extern "C" void airt_test_pool_delete(void *pool) { delete static_cast<FakeDevice *>(pool); }
