// pool.cpp -- kept device memory blocks (declared in xfmm_internal.h).
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <vector>

#include "xfmm_internal.h"

namespace xfmm {
namespace {

constexpr size_t POOL_KEEP = (size_t)2 << 30;       // bytes kept per device
constexpr size_t POOL_MAX_BLOCK = (size_t)512 << 20;  // larger blocks go back to the device at once

struct Kept {
  std::multimap<size_t, void*> blocks;  // by capacity
  size_t bytes = 0;
};
struct Pool {
  std::mutex m;
  std::map<int, Kept> dev;
  std::map<void*, int> owner;  // device of every block handed out
  int holds = 0;
};
// never destroyed: handles may be freed while the process exits
Pool& pool() {
  static Pool* p = new Pool();
  return *p;
}
thread_local int t_quiet = 0;
thread_local bool t_waited = false;

void give_back(Kept& k) {
  for (auto& b : k.blocks) cudaFree(b.second);
  k.blocks.clear();
  k.bytes = 0;
}
}  // namespace

// Capacities in steps of an eighth of a power of two, so that blocks of nearly equal sizes serve each other; the
// exact size for blocks that are never kept (spectra of tens of GB would grow by GBs).
size_t pool_capacity(size_t b) {
  size_t step = 512;
  while (step * 16 < b) step *= 2;
  const size_t r = (b + step - 1) / step * step;
  return r <= POOL_MAX_BLOCK ? r : b;
}

cudaError_t pool_alloc(size_t bytes, void** out, size_t* capacity) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  const size_t want = pool_capacity(bytes);
  Pool& P = pool();
  std::lock_guard<std::mutex> lock(P.m);
  Kept& k = P.dev[dev];
  auto it = k.blocks.lower_bound(want);
  if (it != k.blocks.end() && it->first <= want + want / 4) {
    void* p = it->second;
    *capacity = it->first;
    k.bytes -= it->first;
    k.blocks.erase(it);
    P.owner[p] = dev;
    *out = p;
    return cudaSuccess;
  }
  void* p = nullptr;
  err = cudaMalloc(&p, want);
  if (err == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    give_back(k);
    err = cudaMalloc(&p, want);
  }
  if (err != cudaSuccess) {
    cudaGetLastError();
    return err;
  }
  *capacity = want;
  P.owner[p] = dev;
  *out = p;
  return cudaSuccess;
}

void pool_release(void* p, size_t capacity) noexcept {
  Pool& P = pool();
  int dev = -1, cur = -1;
  bool keep = false;
  {
    std::lock_guard<std::mutex> lock(P.m);
    auto it = P.owner.find(p);
    if (it != P.owner.end()) {
      dev = it->second;
      P.owner.erase(it);
    }
    keep = P.holds > 0 && capacity <= POOL_MAX_BLOCK;
  }
  if (keep && cudaGetDevice(&cur) == cudaSuccess && cur == dev) {
    // no work in flight may still use the block (cudaFree waits in the same way)
    bool idle = t_quiet > 0 && t_waited;
    if (!idle) {
      idle = cudaDeviceSynchronize() == cudaSuccess;
      t_waited = idle;
    }
    if (idle) {
      std::lock_guard<std::mutex> lock(P.m);
      Kept& k = P.dev[dev];
      if (P.holds > 0 && k.bytes + capacity <= POOL_KEEP) {
        k.blocks.emplace(capacity, p);
        k.bytes += capacity;
        return;
      }
    }
  }
  cudaFree(p);
}

void pool_hold() {
  std::lock_guard<std::mutex> lock(pool().m);
  pool().holds++;
}
void pool_unhold() noexcept {
  Pool& P = pool();
  std::lock_guard<std::mutex> lock(P.m);
  if (--P.holds == 0)
    for (auto& d : P.dev) give_back(d.second);
}

PoolQuiet::PoolQuiet() noexcept {
  if (t_quiet++ == 0) t_waited = false;
}
PoolQuiet::~PoolQuiet() {
  if (--t_quiet == 0) t_waited = false;
}

}  // namespace xfmm
