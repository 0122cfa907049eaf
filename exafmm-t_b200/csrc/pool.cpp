// pool.cpp -- kept device memory blocks, and the work that uses them (declared in xfmm_internal.h).
#include <cuda_runtime.h>

#include <algorithm>
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
struct Block {
  int dev;
  uint64_t number;  // of its allocation, ascending
};
struct Pool {
  std::mutex m;
  std::map<int, Kept> dev;
  std::map<void*, Block> owner;  // every block handed out
  uint64_t allocations = 0;
  int holds = 0;
};
// never destroyed: handles may be freed while the process exits
Pool& pool() {
  static Pool* p = new Pool();
  return *p;
}
thread_local UseScope* t_scope = nullptr;  // the API call that this thread is in
thread_local bool t_idle = false;          // an object is being freed and its work is done

// Waits that CUDA allows while another thread captures: of streams and events that take no part in a capture.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
  cudaGetLastError();  // the legacy stream, while a stream that waits for it captures
  return true;
}

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
    P.owner[p] = Block{dev, ++P.allocations};
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
  P.owner[p] = Block{dev, ++P.allocations};
  *out = p;
  return cudaSuccess;
}

void pool_release(void* p, size_t capacity) noexcept {
  Pool& P = pool();
  Block b{-1, 0};
  int cur = -1;
  bool keep = false;
  {
    std::lock_guard<std::mutex> lock(P.m);
    auto it = P.owner.find(p);
    if (it != P.owner.end()) {
      b = it->second;
      P.owner.erase(it);
    }
    keep = P.holds > 0 && capacity <= POOL_MAX_BLOCK;
  }
  if (keep && (t_idle || (t_scope && t_scope->idle(b.number))) && cudaGetDevice(&cur) == cudaSuccess && cur == b.dev) {
    std::lock_guard<std::mutex> lock(P.m);
    Kept& k = P.dev[b.dev];
    if (P.holds > 0 && k.bytes + capacity <= POOL_KEEP) {
      k.blocks.emplace(capacity, p);
      k.bytes += capacity;
      return;
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

bool Uses::wait() const noexcept {
  if (unknown) return false;
  RelaxedCapture relaxed;
  for (const auto& u : last)
    if (cudaEventSynchronize(u.second->e) != cudaSuccess) return false;
  for (const auto& u : graphs)
    if (cudaEventSynchronize(u->e) != cudaSuccess) return false;
  return true;
}

UseScope::UseScope(cudaStream_t s, std::vector<Uses*> objects)
    : s_(s), objects_(std::move(objects)), capturing_(capturing(s)), outer_(t_scope) {
  {
    std::lock_guard<std::mutex> lock(pool().m);
    begin_ = pool().allocations;
  }
  t_scope = this;
}

UseScope::~UseScope() {
  t_scope = outer_;
  if (objects_.empty()) return;
  try {
    unsigned long long id = 0;
    std::shared_ptr<Uses::Event> ev;
    if (capturing_) {
      ev = std::make_shared<Uses::Event>();
      if (cudaEventCreateWithFlags(&ev->e, cudaEventDisableTiming) == cudaSuccess &&
          cudaEventRecordWithFlags(ev->e, s_, cudaEventRecordExternal) == cudaSuccess) {
        for (Uses* u : objects_)
          if (u->graphs.empty() || u->graphs.back() != ev) u->graphs.push_back(ev);
        return;
      }
    }
    bool ok = !capturing_ && cudaStreamGetId(s_, &id) == cudaSuccess;
    // the stream's event of one of the objects, recorded again: all earlier work of the stream is before it
    for (Uses* u : objects_)
      for (auto& l : u->last)
        if (l.first == id) ev = l.second;
    if (ok && !ev) {
      ev = std::make_shared<Uses::Event>();
      ok = cudaEventCreateWithFlags(&ev->e, cudaEventDisableTiming) == cudaSuccess;
    }
    if (ok && cudaEventRecord(ev->e, s_) == cudaSuccess) {
      for (Uses* u : objects_) {
        auto it = std::find_if(u->last.begin(), u->last.end(), [&](const auto& l) { return l.first == id; });
        if (it == u->last.end()) u->last.emplace_back(id, ev);
        else it->second = ev;
      }
      return;
    }
    cudaGetLastError();
  } catch (...) {
  }
  for (Uses* u : objects_) u->unknown = true;
}

bool UseScope::idle(uint64_t allocated) const noexcept {
  if (capturing_) return false;
  RelaxedCapture relaxed;
  if (cudaStreamSynchronize(s_) != cudaSuccess) return false;
  if (allocated > begin_) return true;
  for (const Uses* u : objects_)
    if (!u->wait()) return false;
  return true;
}

FreeScope::FreeScope(const Uses& u) noexcept { t_idle = u.wait(); }
FreeScope::~FreeScope() { t_idle = false; }

}  // namespace xfmm
