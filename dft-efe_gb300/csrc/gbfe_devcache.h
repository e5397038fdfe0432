// gbfe_devcache.h -- device blocks kept for reuse between calls.
//
// cudaFree synchronises the device, so temporaries that come and go with every call
// (and a server's requests) are parked instead and reused by exact size.  A block is
// parked in the scope of the call that frees it, and goes to the cache, where any
// scope of that cache may take it, once the owner has synchronised the streams that
// may still use it.  Several threads may work with one cache.  When an allocation
// fails, the blocks that the failing call has parked (cudaFree waits for their last
// use) and those of every cache in the process are given back before it is tried
// again: a program gets the memory it would have without caches.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <set>
#include <utility>
#include <vector>

namespace gbfe {

using DevBlocks = std::vector<std::pair<size_t, void *>>;

class DevCache {
 public:
  DevCache() {
    std::lock_guard<std::mutex> lk(all().mu);
    all().caches.insert(this);
  }
  ~DevCache() {
    {
      std::lock_guard<std::mutex> lk(all().mu);
      all().caches.erase(this);
    }
    release();
  }
  DevCache(const DevCache &) = delete;
  DevCache &operator=(const DevCache &) = delete;
  bool take(size_t bytes, void **p) {
    std::lock_guard<std::mutex> lk(mu_);
    auto it = ready_.find(bytes);
    if (it == ready_.end()) return false;
    *p = it->second;
    held_ -= bytes;
    ready_.erase(it);
    return true;
  }
  // takes the blocks over as far as they fit under cap bytes and frees the others
  void put(DevBlocks &blocks, size_t cap) {
    DevBlocks over;
    {
      std::lock_guard<std::mutex> lk(mu_);
      for (auto &b : blocks) {
        if (held_ + b.first > cap) {
          over.push_back(b);
          continue;
        }
        ready_.insert(b);
        held_ += b.first;
      }
    }
    for (auto &b : over) cudaFree(b.second);
    blocks.clear();
  }
  size_t bytes() const {
    std::lock_guard<std::mutex> lk(mu_);
    return held_;
  }
  void release() {
    std::multimap<size_t, void *> out;
    {
      std::lock_guard<std::mutex> lk(mu_);
      out.swap(ready_);
      held_ = 0;
    }
    for (auto &b : out) cudaFree(b.second);
  }
  static void release_all() {
    std::lock_guard<std::mutex> lk(all().mu);
    for (DevCache *c : all().caches) c->release();
  }

 private:
  struct All {
    std::mutex mu;
    std::set<DevCache *> caches;
  };
  static All &all() {
    static All *a = new All;  // (outlives caches of static objects)
    return *a;
  }
  mutable std::mutex mu_;
  std::multimap<size_t, void *> ready_;
  size_t held_ = 0;
};

// What a thread has freed since the streams were last synchronised; with the blocks
// of the cache at most cap bytes (past it a free goes to cudaFree).
struct DevScope {
  DevCache &cache;
  size_t cap;
  DevBlocks parked = {};
  size_t parked_bytes = 0;
  bool refused = false;  // a block did not fit
  void mark_safe() {
    cache.put(parked, cap);
    parked_bytes = 0;
  }
  void free_parked() {
    for (auto &b : parked) cudaFree(b.second);
    parked.clear();
    parked_bytes = 0;
  }
};
inline DevScope *&thread_dev_scope() {
  static thread_local DevScope *scope = nullptr;
  return scope;
}

inline cudaError_t dev_alloc(void **p, size_t bytes) {
  DevScope *s = thread_dev_scope();
  if (s && s->cache.take(bytes, p)) return cudaSuccess;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    (void)cudaGetLastError();
    if (s) s->free_parked();
    DevCache::release_all();
    e = cudaMalloc(p, bytes);
  }
  return e;
}
inline void dev_free(void *p, size_t bytes) {
  DevScope *s = thread_dev_scope();
  if (s && s->parked_bytes + s->cache.bytes() + bytes <= s->cap) {
    s->parked.emplace_back(bytes, p);
    s->parked_bytes += bytes;
    return;
  }
  if (s) s->refused = true;
  cudaFree(p);
}

}  // namespace gbfe
