// dev_pool.h -- device memory of plans that are gone, for the next plan.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <map>
#include <mutex>
#include <new>

// The one-shot calls (advance_native, advance_fortran, the torch op) build a
// plan per call, and its allocations and frees took most of it: 0.8 of 0.93 ms
// at 2,592 columns, where the step takes 0.14.  A context and its plans share
// one pool; it holds at most kLimit bytes and gives everything back with the
// last of them, and before an allocation of the context fails.  A block comes
// back only once the device has finished with it (give and build_tiles
// synchronise first, as cudaFree did), so any stream may use it next; where the
// device cannot be waited for (a stream is being captured), it is set aside
// until a later wait has succeeded.  The mutex makes the pool safe from several
// host threads.  No call throws.
class DevPool {
 public:
  static constexpr size_t kLimit = size_t(256) << 20;

  explicit DevPool(int device) : device_(device) {}
  ~DevPool() {
    int was = 0;
    const bool ok = cudaGetDevice(&was) == cudaSuccess && cudaSetDevice(device_) == cudaSuccess;
    for (auto& b : blocks_)
      if (b.second.state != kUsed) cudaFree(b.first);
    if (ok) cudaSetDevice(was);
  }
  DevPool(const DevPool&) = delete;
  DevPool& operator=(const DevPool&) = delete;

  cudaError_t get(void** p, size_t bytes) {
    bytes = (std::max<size_t>(bytes, 1) + 511) & ~size_t(511);
    std::lock_guard<std::mutex> lock(mu_);
    // the smallest free block that fits, and wastes no more than half or 64 KB
    auto best = blocks_.end();
    for (auto it = blocks_.begin(); it != blocks_.end(); ++it) {
      const Block& b = it->second;
      if (b.state == kFree && b.bytes >= bytes && b.bytes <= std::max(2 * bytes, size_t(64) << 10) &&
          (best == blocks_.end() || b.bytes < best->second.bytes))
        best = it;
    }
    if (best != blocks_.end()) {
      best->second.state = kUsed;
      held_ -= best->second.bytes;
      *p = best->first;
      return cudaSuccess;
    }
    const cudaError_t e = take(p, bytes);
    if (e != cudaSuccess) return e;
    try {
      blocks_[*p] = Block{bytes, kUsed, 0};
    } catch (const std::bad_alloc&) {
      cudaFree(*p);
      return cudaErrorMemoryAllocation;
    }
    return e;
  }

  // Memory that is not the pool's (the caller frees it), with what the pool
  // holds given back first where it would not fit.
  cudaError_t outside(void** p, size_t bytes) {
    std::lock_guard<std::mutex> lock(mu_);
    return take(p, bytes);
  }

  // Waits for everything launched on the pool's device, as cudaFree does, and
  // takes back blocks of get() (or NULL) that only work launched so far uses.
  void give(std::initializer_list<void*> blocks) {
    uint64_t upto = 0;
    {
      std::lock_guard<std::mutex> lock(mu_);
      upto = ++turn_;
      for (void* p : blocks) {
        auto it = blocks_.find(p);
        if (it == blocks_.end()) continue;
        it->second.state = kAside;
        it->second.turn = upto;
      }
    }
    int was = 0;
    const bool ok = cudaGetDevice(&was) == cudaSuccess && cudaSetDevice(device_) == cudaSuccess;
    if (cudaDeviceSynchronize() == cudaSuccess) {
      // what was set aside before this wait began, by any thread
      std::lock_guard<std::mutex> lock(mu_);
      for (auto it = blocks_.begin(); it != blocks_.end();) {
        auto at = it++;
        if (at->second.state == kAside && at->second.turn <= upto) keep(at);
      }
    } else {
      cudaGetLastError();
    }
    if (ok) cudaSetDevice(was);
  }

  // p: a block of get() that nothing on the device uses any more, or NULL
  void put(void* p) {
    std::lock_guard<std::mutex> lock(mu_);
    auto it = blocks_.find(p);
    if (it != blocks_.end()) keep(it);
  }

 private:
  enum State { kUsed, kAside, kFree };  // given out; given back, but perhaps still in use; for the next plan
  struct Block {
    size_t bytes;
    State state;
    uint64_t turn;  // the give() that set it aside
  };

  void keep(std::map<void*, Block>::iterator it) {
    if (held_ + it->second.bytes <= kLimit) {
      it->second.state = kFree;
      held_ += it->second.bytes;
    } else {
      cudaFree(it->first);
      blocks_.erase(it);
    }
  }
  cudaError_t take(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    for (auto it = blocks_.begin(); it != blocks_.end();) {
      auto at = it++;
      if (at->second.state != kFree) continue;
      cudaFree(at->first);
      blocks_.erase(at);
    }
    held_ = 0;
    return cudaMalloc(p, bytes);
  }

  const int device_;
  std::mutex mu_;
  std::map<void*, Block> blocks_;
  size_t held_ = 0;  // bytes of the free ones
  uint64_t turn_ = 0;
};
