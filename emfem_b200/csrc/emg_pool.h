// Device memory that contexts have freed, kept for the next allocations
// (emg_pool.cpp).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <vector>

namespace emg {

struct DevicePool;

// A context as the pool sees it.  Its work runs on one stream, so a block that
// it has freed can go straight back to it without waiting for the GPU.  Other
// contexts get the block once that stream has been seen idle (settle()).
struct PoolUser {
  DevicePool *pool = nullptr;
  cudaStream_t stream = nullptr;
  bool unsettled = false;  // has freed blocks since the last settle()
  uint64_t settled = 0;    // its blocks up to this tick may serve others
  PoolUser() = default;
  PoolUser(const PoolUser &) = delete;
  PoolUser &operator=(const PoolUser &) = delete;
  void join(DevicePool &p, cudaStream_t s);
  ~PoolUser();  // gives its blocks back
};

// One per device and process, shared by its contexts and safe with several
// threads.  Above 1 MB cudaMalloc and cudaFree take 0.3 ms each, below it as
// much where the driver's slab of 2 MB is full or falls empty; an AMS setup
// needs some 150 of them.  Kept at most: 4 GB, and an eighth of the memory
// that is free with it once more than 256 MB are kept; the blocks that have
// lain longest go first.  A user's blocks are given back when its linear system
// or it is destroyed or its mesh is set, everything when an allocation fails.
struct DevicePool {
  static constexpr size_t kKeep = size_t(4) << 30, kAsk = size_t(256) << 20;
  struct Block {
    void *p;
    PoolUser *owner;
    uint64_t tick;
  };
  static DevicePool &of(int device);
  void *get(size_t &bytes, PoolUser *u);  // at least `bytes` (set to the block's size); null when out of memory
  void put(void *p, size_t bytes, PoolUser *u);
  void settle(PoolUser *u);  // nothing of u's stream is running or queued
  void trim(PoolUser *u);
  size_t cached();
  std::atomic<int> users{0};

 private:
  std::mutex mu;
  std::multimap<size_t, Block> blocks;  // by size
  size_t kept = 0, limit = kKeep;
  uint64_t clock = 0;
  std::chrono::steady_clock::time_point asked{};
  void evict(std::vector<void *> &out);  // down to the limit, under the lock
  void ask_free();                       // sets the limit by the memory that is free
};

// the user whose pool allocations of this thread come from (null: cudaMalloc)
PoolUser *&current_user();
struct PoolScope {
  PoolUser *before;
  explicit PoolScope(PoolUser &u) : before(current_user()) { current_user() = &u; }
  PoolScope(const PoolScope &) = delete;
  PoolScope &operator=(const PoolScope &) = delete;
  ~PoolScope();  // settles the user where its stream is idle and others might want its blocks
};

}  // namespace emg
