// Device and pinned host memory of systems, kept for reuse while systems or a
// scene server are alive. Building and destroying a system takes some fifty
// buffers, and cudaMalloc / cudaFree (which waits for the whole device) took
// most of that time: a served batch of six scenes spent 70 to 160 ms, of which
// its steps are about 20.
//
// A freed block is kept by its size class (an eighth of a power of two) and
// handed out again by whichever thread asks first; the owner of a block frees it
// only when no stream uses it any more. At most kKeep bytes per device (and
// kKeepHost pinned) are kept; what is beyond goes back to the driver at once, and
// everything does when the last holder (PoolUse) is gone or an allocation fails.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

#include "sph_host.hpp"

namespace sph {

class Pool {
 public:
  static constexpr size_t kKeep = (size_t)1 << 30;
  static constexpr size_t kKeepHost = (size_t)64 << 20;
  static constexpr int kHost = -1;  // "device" of pinned host memory

  static Pool& get() {
    static Pool* p = new Pool;  // never destroyed: buffers may outlive static destructors
    return *p;
  }

  // `bytes` of memory of the current device, or pinned memory (where = kHost).
  void* alloc(size_t bytes, int where) {
    const size_t size = size_class(bytes);
    {
      std::lock_guard<std::mutex> lock(mu_);
      Kept& k = kept_[where];
      auto it = k.blocks.find(size);
      if (it != k.blocks.end() && !it->second.empty()) {
        void* p = it->second.back();
        it->second.pop_back();
        k.bytes -= size;
        sizes_[p] = {where, size};
        return p;
      }
    }
    void* p = nullptr;
    cudaError_t e = raw_alloc(&p, size, where);
    if (e == cudaErrorMemoryAllocation) {  // what is kept may be what is missing
      cudaGetLastError();
      trim();
      e = raw_alloc(&p, size, where);
    }
    if (e != cudaSuccess) cudaGetLastError();
    cuda_check(e, where == kHost ? "cudaMallocHost" : "cudaMalloc");
    std::lock_guard<std::mutex> lock(mu_);
    sizes_[p] = {where, size};
    return p;
  }

  // The caller has made sure that no stream uses the block.
  void free(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lock(mu_);
    const auto it = sizes_.find(p);
    const Block b = it->second;
    sizes_.erase(it);
    Kept& k = kept_[b.where];
    if (users_ > 0 && k.bytes + b.size <= (b.where == kHost ? kKeepHost : kKeep)) {
      k.blocks[b.size].push_back(p);
      k.bytes += b.size;
    } else {
      raw_free(p, b.where);
    }
  }

  void hold() {
    std::lock_guard<std::mutex> lock(mu_);
    ++users_;
  }
  void release() {
    bool last;
    {
      std::lock_guard<std::mutex> lock(mu_);
      last = --users_ == 0;
    }
    if (last) trim();
  }

  // Gives everything kept back to the driver, or what is kept of one device.
  void trim() { trim_if([](int) { return true; }); }
  void trim(int where) { trim_if([where](int w) { return w == where; }); }

  size_t kept_bytes(int where) {
    std::lock_guard<std::mutex> lock(mu_);
    return kept_[where].bytes;
  }

 private:
  template <class F>
  void trim_if(F&& of) {
    std::lock_guard<std::mutex> lock(mu_);
    for (auto& k : kept_) {
      if (!of(k.first)) continue;
      for (auto& c : k.second.blocks)
        for (void* p : c.second) raw_free(p, k.first);
      k.second.blocks.clear();
      k.second.bytes = 0;
    }
  }

  struct Kept {
    std::map<size_t, std::vector<void*>> blocks;
    size_t bytes = 0;
  };
  struct Block {
    int where;
    size_t size;
  };
  std::mutex mu_;
  std::map<int, Kept> kept_;
  std::map<void*, Block> sizes_;
  int users_ = 0;

  static size_t size_class(size_t bytes) {
    size_t step = 512;
    while (step * 16 <= bytes) step *= 2;  // bytes in [8 step, 16 step): a class per step
    return (bytes + step - 1) / step * step;
  }
  static cudaError_t raw_alloc(void** p, size_t size, int where) {
    return where == kHost ? cudaMallocHost(p, size) : cudaMalloc(p, size);
  }
  // (a device pointer may be freed with any device current)
  static void raw_free(void* p, int where) {
    if (where == kHost) cudaFreeHost(p);
    else cudaFree(p);
  }
};

// Keeps the pool's memory while it lives.
struct PoolUse {
  PoolUse() { Pool::get().hold(); }
  ~PoolUse() { Pool::get().release(); }
  PoolUse(const PoolUse&) = delete;
  PoolUse& operator=(const PoolUse&) = delete;
};

}  // namespace sph
