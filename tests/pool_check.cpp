// Device memory pool (emg_pool.cpp) against a counting stand-in for the CUDA
// calls it makes, built and run by test_pool_host_cpu.py: what is kept is
// bounded and the blocks that have lain longest go first, a block goes to
// another context only once its owner's stream has been idle, a failing
// allocation gets everything that is kept, little is kept where little is free,
// a context gives its blocks back, and threads may use it at once.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <set>
#include <thread>

#include "emg_pool.h"

using namespace emg;

static std::mutex mu;
static std::map<void *, size_t> live;
static std::set<void *> freed;
static size_t in_use = 0, device_bytes = size_t(64) << 30;
static bool busy = false;
static uintptr_t next_address = 4096;
static std::atomic<long> mallocs{0};

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
  std::lock_guard<std::mutex> lock(mu);
  ++mallocs;
  if (in_use + n > device_bytes) return cudaErrorMemoryAllocation;
  *p = reinterpret_cast<void *>(next_address);
  next_address += (n + 4095) / 4096 * 4096;
  live[*p] = n;
  in_use += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> lock(mu);
  auto it = live.find(p);
  if (it == live.end()) {
    std::printf("free of an unknown block\n");
    std::exit(1);
  }
  in_use -= it->second;
  live.erase(it);
  freed.insert(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  std::lock_guard<std::mutex> lock(mu);
  *f = device_bytes - in_use;
  *t = device_bytes;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return busy ? cudaErrorNotReady : cudaSuccess; }
}

#define CHECK(x)                                          \
  do {                                                    \
    if (!(x)) {                                           \
      std::printf("line %d: %s\n", __LINE__, #x);         \
      return 1;                                           \
    }                                                     \
  } while (0)

static const size_t MB = size_t(1) << 20;

int main() {
  DevicePool &pool = DevicePool::of(0);
  CHECK(&pool == &DevicePool::of(0) && &pool != &DevicePool::of(1));
  {  // sizes that change from round to round: the newest stay, the oldest go
    PoolUser u;
    u.join(pool, nullptr);
    const size_t step = 300 * MB;
    void *last = nullptr;
    for (int round = 0; round < 40; ++round) {
      size_t n = step + (size_t)round * 64 * MB;  // never within an eighth of a smaller kept one
      void *p = pool.get(n, &u);
      CHECK(p);
      pool.put(p, n, &u);
      CHECK(pool.cached() <= DevicePool::kKeep);
      CHECK(in_use == pool.cached());
      last = p;
    }
    CHECK(pool.cached() > 0);
    size_t n = step + 39 * 64 * MB;
    const long m0 = mallocs;
    CHECK(pool.get(n, &u) == last && mallocs == m0);  // the last size is there
    pool.put(last, n, &u);
    size_t big = DevicePool::kKeep + MB;  // larger than all that may be kept
    void *p = pool.get(big, &u);
    CHECK(p);
    pool.put(p, big, &u);
    CHECK(pool.cached() <= DevicePool::kKeep && freed.count(p));
  }
  CHECK(pool.cached() == 0 && in_use == 0);  // the user is gone
  {  // another context, before and after the owner's stream was seen idle
    PoolUser a, b;
    a.join(pool, nullptr);
    b.join(pool, nullptr);
    size_t n = 2 * MB;
    void *p = pool.get(n, &a);
    busy = true;
    {
      const PoolScope on(a);
      CHECK(current_user() == &a);
      pool.put(p, n, &a);
    }
    CHECK(current_user() == nullptr);
    void *q = pool.get(n, &b);
    CHECK(q != p);
    CHECK(pool.get(n, &a) == p);  // its own needs no wait
    busy = false;
    {
      const PoolScope on(a);
      pool.put(p, n, &a);
    }
    CHECK(pool.get(n, &b) == p);
    pool.put(p, n, &b);
    pool.put(q, n, &b);
    pool.trim(&a);
    CHECK(pool.cached() == 2 * n);  // the blocks are b's now
    pool.trim(&b);
    CHECK(pool.cached() == 0 && in_use == 0);
  }
  {  // a full device: an allocation gets what other contexts keep, then fails
    PoolUser a, b;
    a.join(pool, nullptr);
    b.join(pool, nullptr);
    device_bytes = 1024 * MB;
    size_t n = 700 * MB;
    void *p = pool.get(n, &a);
    pool.put(p, n, &a);
    size_t m = 800 * MB;
    void *q = pool.get(m, &b);
    CHECK(q && pool.cached() == 0);
    size_t k = 300 * MB;
    CHECK(!pool.get(k, &a));
    pool.put(q, m, &b);
  }
  CHECK(in_use == 0);
  {  // little memory free: an eighth of it is kept, at least 256 MB
    PoolUser a;
    a.join(pool, nullptr);
    device_bytes = 4096 * MB;
    void *p[8];
    size_t n = 400 * MB;
    std::this_thread::sleep_for(std::chrono::milliseconds(150));  // it asks ten times a second at most
    for (void *&x : p) x = pool.get(n, &a);
    for (void *x : p) pool.put(x, n, &a);
    CHECK(pool.cached() <= 512 * MB);
    device_bytes = size_t(64) << 30;
    std::this_thread::sleep_for(std::chrono::milliseconds(150));
    for (void *&x : p) x = pool.get(n, &a);
    for (void *x : p) pool.put(x, n, &a);
    CHECK(pool.cached() == 8 * n);  // and more again where much is free
  }
  CHECK(in_use == 0);
  {  // threads, each with its context
    std::atomic<int> bad{0};
    std::vector<std::thread> th;
    for (int t = 0; t < 8; ++t)
      th.emplace_back([&, t] {
        PoolUser u;
        u.join(pool, nullptr);
        for (int i = 0; i < 2000; ++i) {
          const PoolScope on(u);
          size_t n = (size_t)(1 + (i * 7 + t) % 50) * 100000;
          void *p = pool.get(n, &u);
          if (!p) ++bad;
          else pool.put(p, n, &u);
          if (i % 500 == 499) pool.trim(&u);
        }
      });
    for (auto &x : th) x.join();
    CHECK(bad == 0);
  }
  CHECK(pool.cached() == 0 && in_use == 0 && live.empty() && pool.users == 0);
  std::printf("ok\n");
  return 0;
}
