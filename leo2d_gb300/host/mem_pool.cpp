// mem_pool.cpp - released device memory kept for the next allocations (csrc/mem_pool.h).
#include "leo2d_gb300/csrc/mem_pool.h"

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

namespace leo2d {

namespace {

struct KeptBlock {
  void* p;
  size_t bytes;
  const MemPool* owner;  // the context whose stream may still use it; null: anyone's
};

// What the process keeps of one device, oldest first.
struct DeviceKept {
  std::vector<KeptBlock> blocks;
  size_t bytes = 0;
  int contexts = 0;
};

// All of it, under one lock.
struct Kept {
  std::mutex mu;
  std::map<int, DeviceKept> devices;
};
Kept& kept_state() {
  static Kept* k = new Kept();  // outlives every pool
  return *k;
}
constexpr size_t kMaxBlocks = 1024;  // of a device

void drop_block(DeviceKept& k, size_t i) {
  cudaFree(k.blocks[i].p);  // waits for work that still uses it
  k.bytes -= k.blocks[i].bytes;
  k.blocks.erase(k.blocks.begin() + (std::ptrdiff_t)i);
}

}  // namespace

MemPool::MemPool(int device, cudaStream_t stream, size_t device_bytes)
    : device_(device), stream_(stream), cap_(std::min(device_bytes / 16, (size_t)16 << 30)) {
  Kept& k = kept_state();
  std::lock_guard<std::mutex> lock(k.mu);
  ++k.devices[device_].contexts;
}

MemPool::~MemPool() { close(); }

void MemPool::enter() {
  std::lock_guard<std::mutex> lock(kept_state().mu);
  ++depth_;
}

void MemPool::leave() {
  Kept& all = kept_state();
  std::lock_guard<std::mutex> lock(all.mu);
  if (--depth_ != 0 || closed_) return;
  DeviceKept& k = all.devices[device_];
  bool mine = false;
  for (const KeptBlock& b : k.blocks) mine |= b.owner == this;
  if (!mine) return;
  if (cudaStreamQuery(stream_) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  for (KeptBlock& b : k.blocks)
    if (b.owner == this) b.owner = nullptr;
}

// The smallest block of at least `bytes` and at most a quarter (or 64 KB) more.
void* MemPool::take(size_t bytes, size_t* got) {
  Kept& all = kept_state();
  std::lock_guard<std::mutex> lock(all.mu);
  DeviceKept& k = all.devices[device_];
  size_t best = k.blocks.size();
  const size_t most = bytes + std::max(bytes / 4, (size_t)64 << 10);
  for (size_t i = 0; i < k.blocks.size(); ++i) {
    const KeptBlock& b = k.blocks[i];
    if ((!b.owner || b.owner == this) && b.bytes >= bytes && b.bytes <= most &&
        (best == k.blocks.size() || b.bytes < k.blocks[best].bytes))
      best = i;
  }
  if (best == k.blocks.size()) return nullptr;
  const KeptBlock b = k.blocks[best];
  k.blocks.erase(k.blocks.begin() + (std::ptrdiff_t)best);
  k.bytes -= b.bytes;
  *got = b.bytes;
  return b.p;
}

bool MemPool::give(void* p, size_t bytes) {
  Kept& all = kept_state();
  std::lock_guard<std::mutex> lock(all.mu);
  if (closed_ || bytes > cap_) return false;
  DeviceKept& k = all.devices[device_];
  const MemPool* owner = this;
  if (depth_ == 0) {  // outside any call: anyone's once the stream is idle
    if (cudaStreamQuery(stream_) == cudaSuccess) owner = nullptr;
    else cudaGetLastError();
  }
  while (!k.blocks.empty() && (k.bytes + bytes > cap_ || k.blocks.size() >= kMaxBlocks)) drop_block(k, 0);
  try {
    k.blocks.push_back(KeptBlock{p, bytes, owner});
  } catch (...) {
    return false;
  }
  k.bytes += bytes;
  return true;
}

void MemPool::close() {
  Kept& all = kept_state();
  std::lock_guard<std::mutex> lock(all.mu);
  if (closed_) return;
  closed_ = true;
  DeviceKept& k = all.devices[device_];
  --k.contexts;
  for (size_t i = k.blocks.size(); i-- > 0;)
    if (k.blocks[i].owner == this || k.contexts == 0) drop_block(k, i);
}

size_t MemPool::kept(int device) {
  Kept& all = kept_state();
  std::lock_guard<std::mutex> lock(all.mu);
  return all.devices[device].bytes;
}

void MemPool::flush(int device) {
  Kept& all = kept_state();
  std::lock_guard<std::mutex> lock(all.mu);
  DeviceKept& k = all.devices[device];
  while (!k.blocks.empty()) drop_block(k, k.blocks.size() - 1);
}

cudaError_t device_malloc(void** p, size_t bytes, size_t* got) {
  cudaError_t e = cudaMalloc(p, *got);
  int device = 0;
  if (e == cudaErrorMemoryAllocation && cudaGetDevice(&device) == cudaSuccess && MemPool::kept(device) != 0) {
    cudaGetLastError();
    MemPool::flush(device);
    e = cudaMalloc(p, *got);
  }
  if (e == cudaErrorMemoryAllocation && *got > bytes) {
    cudaGetLastError();
    *got = bytes;
    e = cudaMalloc(p, *got);
  }
  // (the status says it; left behind, it would be taken for a failed launch of what runs next)
  if (e == cudaErrorMemoryAllocation) cudaGetLastError();
  return e;
}

}  // namespace leo2d
