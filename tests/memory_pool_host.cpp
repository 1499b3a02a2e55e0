// Checks of host/mem_pool.cpp against a CUDA runtime of two small devices, made here:
// every allocation and release is counted, and nothing needs a GPU.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "leo2d_gb300/csrc/mem_pool.h"

using leo2d::MemPool;

static const size_t MB = (size_t)1 << 20;
static int g_current = 0;
static size_t g_free[2] = {512 * MB, 512 * MB};
static std::map<void*, std::pair<int, size_t>> g_live;
static int g_busy = 0;  // streams still run
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = g_current; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (n > g_free[g_current]) return g_last = cudaErrorMemoryAllocation;
  *p = std::malloc(1);
  g_live[*p] = {g_current, n};
  g_free[g_current] -= n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  auto it = g_live.find(p);
  if (it == g_live.end()) std::abort();
  g_free[it->second.first] += it->second.second;
  g_live.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t) { return g_busy ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
}

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return __LINE__; } } while (0)

static void* make(int device, size_t n) {
  g_current = device;
  void* p = nullptr;
  size_t got = n;
  return leo2d::device_malloc(&p, n, &got) == cudaSuccess ? p : nullptr;
}

int main() {
  {
    MemPool a(0, nullptr, 16 * 256 * MB), b(1, nullptr, 16 * 256 * MB), c(0, nullptr, 16 * 256 * MB);
    // what is kept of one device is not counted for, nor taken by, the other
    void* p = make(0, 100 * MB);
    CHECK(a.give(p, 100 * MB));
    CHECK(MemPool::kept(0) == 100 * MB && MemPool::kept(1) == 0);
    size_t got = 0;
    CHECK(b.take(100 * MB, &got) == nullptr);
    // an allocation that does not fit gives back its own device's blocks only
    void* q = make(1, 200 * MB);
    CHECK(b.give(q, 200 * MB));
    void* big = make(1, 500 * MB);
    CHECK(big && MemPool::kept(1) == 0 && MemPool::kept(0) == 100 * MB);
    cudaFree(big);
    CHECK(make(1, 600 * MB) == nullptr && MemPool::kept(0) == 100 * MB);
    // the bound is each device's: 256 MB here, oldest first out
    void* r = make(1, 256 * MB);
    CHECK(b.give(r, 256 * MB) && MemPool::kept(0) == 100 * MB && MemPool::kept(1) == 256 * MB);
    void* s = make(0, 200 * MB);
    CHECK(a.give(s, 200 * MB) && MemPool::kept(0) == 200 * MB && MemPool::kept(1) == 256 * MB);
    // a block released while its stream runs is its own context's until the call ends
    void* t = make(0, 40 * MB);
    g_busy = 1;
    c.enter();
    CHECK(c.give(t, 40 * MB));
    CHECK(a.take(40 * MB, &got) == nullptr);
    g_busy = 0;
    c.leave();
    CHECK(a.take(40 * MB, &got) == t && got == 40 * MB);
    cudaFree(t);
    // the last context of a device gives its blocks back, whatever another device keeps
    b.close();
    CHECK(MemPool::kept(1) == 0 && MemPool::kept(0) == 200 * MB);
    MemPool::flush(0);
    CHECK(MemPool::kept(0) == 0);
  }
  {
    // an allocation whose rounded size does not fit, but itself does
    MemPool a(0, nullptr, 16 * 256 * MB);
    void *p = make(0, 100 * MB), *q = nullptr;
    CHECK(a.give(p, 100 * MB));
    size_t got = 544 * MB;
    CHECK(leo2d::device_malloc(&q, 510 * MB, &got) == cudaSuccess && got == 510 * MB && g_free[0] == 2 * MB);
    cudaFree(q);
    got = 512 * MB;
    CHECK(leo2d::device_malloc(&q, 510 * MB, &got) == cudaSuccess && got == 512 * MB);
    cudaFree(q);
    got = 544 * MB;
    CHECK(leo2d::device_malloc(&q, 513 * MB, &got) == cudaErrorMemoryAllocation);
    CHECK(cudaGetLastError() == cudaSuccess);  // nothing left for the next launch's check
  }
  CHECK(g_live.empty() && g_free[0] == 512 * MB && g_free[1] == 512 * MB);
  return 0;
}
