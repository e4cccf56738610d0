// Device memory pool shared by the contexts of a process.

#include "emg_pool.h"

#include <algorithm>

namespace emg {

PoolUser *&current_user() {
  static thread_local PoolUser *u = nullptr;
  return u;
}

void PoolUser::join(DevicePool &p, cudaStream_t s) {
  pool = &p;
  stream = s;
  ++p.users;
}

PoolUser::~PoolUser() {
  if (!pool) return;
  pool->trim(this);
  --pool->users;
}

PoolScope::~PoolScope() {
  PoolUser *u = current_user();
  current_user() = before;
  if (!u->unsettled || u->pool->users < 2) return;
  const cudaError_t e = cudaStreamQuery(u->stream);
  if (e == cudaSuccess) u->pool->settle(u);
  else if (e == cudaErrorNotReady) (void)cudaGetLastError();
}

DevicePool &DevicePool::of(int device) {
  static std::mutex mu;
  static auto *pools = new std::map<int, DevicePool>;  // contexts may outlive static objects
  std::lock_guard<std::mutex> lock(mu);
  return (*pools)[device];
}

void DevicePool::evict(std::vector<void *> &out) {
  while (kept > limit && !blocks.empty()) {
    auto old = std::min_element(blocks.begin(), blocks.end(),
                                [](const auto &a, const auto &b) { return a.second.tick < b.second.tick; });
    out.push_back(old->second.p);
    kept -= old->first;
    blocks.erase(old);
  }
}

// cudaFree waits for the GPU, so a block may go back whoever used it last
static void give_back(const std::vector<void *> &v) {
  for (void *p : v) cudaFree(p);
}

void *DevicePool::get(size_t &bytes, PoolUser *u) {
  bytes = (bytes + 511) / 512 * 512;
  {
    std::lock_guard<std::mutex> lock(mu);
    // a block up to an eighth (and 64 KB) larger than asked for
    const size_t most = bytes + bytes / 8 + 65536;
    for (auto it = blocks.lower_bound(bytes); it != blocks.end() && it->first <= most; ++it)
      if (it->second.owner == u || it->second.tick <= it->second.owner->settled) {
        void *p = it->second.p;
        bytes = it->first;
        kept -= bytes;
        blocks.erase(it);
        return p;
      }
  }
  void *p = nullptr;
  if (cudaMalloc(&p, bytes) == cudaSuccess) return p;
  (void)cudaGetLastError();
  std::vector<void *> all;
  {
    std::lock_guard<std::mutex> lock(mu);
    for (auto &b : blocks) all.push_back(b.second.p);
    blocks.clear();
    kept = 0;
  }
  give_back(all);
  if (!all.empty() && cudaMalloc(&p, bytes) == cudaSuccess) return p;
  (void)cudaGetLastError();
  return nullptr;
}

void DevicePool::put(void *p, size_t bytes, PoolUser *u) {
  std::vector<void *> out;
  bool ask = false;
  try {
    std::lock_guard<std::mutex> lock(mu);
    blocks.emplace(bytes, Block{p, u, ++clock});
    kept += bytes;
    u->unsettled = true;
    p = nullptr;
    if (kept > kAsk) {  // at most ten times a second: the question takes longer than a small call
      const auto now = std::chrono::steady_clock::now();
      ask = now - asked > std::chrono::milliseconds(100);
      if (ask) asked = now;
    }
    if (!ask) evict(out);
  } catch (...) {  // no host memory for the entry, or for the list of those to go
    if (p) cudaFree(p);
  }
  give_back(out);
  if (ask) ask_free();
}

void DevicePool::ask_free() {
  size_t free = 0, total = 0;
  if (cudaMemGetInfo(&free, &total) != cudaSuccess) (void)cudaGetLastError();
  std::vector<void *> out;
  try {
    std::lock_guard<std::mutex> lock(mu);
    limit = std::max(kAsk, std::min(kKeep, (free + kept) / 8));
    evict(out);
  } catch (...) {
  }
  give_back(out);
}

void DevicePool::settle(PoolUser *u) {
  std::lock_guard<std::mutex> lock(mu);
  u->settled = clock;
  u->unsettled = false;
}

void DevicePool::trim(PoolUser *u) {
  std::vector<void *> out;
  {
    std::lock_guard<std::mutex> lock(mu);
    for (auto it = blocks.begin(); it != blocks.end();)
      if (it->second.owner == u) {
        out.push_back(it->second.p);
        kept -= it->first;
        it = blocks.erase(it);
      } else {
        ++it;
      }
    u->unsettled = false;
  }
  give_back(out);
}

size_t DevicePool::cached() {
  std::lock_guard<std::mutex> lock(mu);
  return kept;
}

}  // namespace emg
