// mem_pool.h - device memory kept between calls (host code; host/mem_pool.cpp).
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>

namespace leo2d {

// Released device memory, kept for the next allocations. Mapping and unmapping the
// arrays of a job took 14 of its 122 ms (2.4M orbitals) and 8 of the 46 ms of a Kubo
// trace; of a 76-orbital k point's 2.8 ms, 0.2.
//
// Order: a context runs everything on its one stream, so a block that a call releases
// while kernels still use it may serve the same context's next allocation (its
// pending blocks). When no call runs on the context and its stream is idle, they pass
// to the blocks that every context of the device may take. A buffer goes back through
// the context that made it, inside a call on that context or outside any call (calls
// synchronise before they return, also when they fail); one released inside a call on
// another context is freed with cudaFree, which waits.
// Bounds: what the process keeps of a device is at most 16 GiB or a sixteenth of the
// device's memory, whichever is less, oldest first out; an allocation that fails
// gives back what is kept of its device and tries again, and closing the last context
// of a device gives it back too.
// Thread-safe.
class MemPool {
 public:
  MemPool(int device, cudaStream_t stream, size_t device_bytes);
  ~MemPool();
  void enter();  // a call on the context begins / ends (calls nest)
  void leave();
  void* take(size_t bytes, size_t* got);  // null: nothing fits
  bool give(void* p, size_t bytes);       // false: not kept, the caller frees it
  void close();                           // the context goes: keeps nothing more
  static size_t kept(int device);         // bytes kept of a device
  static void flush(int device);          // gives them back
 private:
  int device_, depth_ = 0;
  cudaStream_t stream_;
  size_t cap_;
  bool closed_ = false;
};

// cudaMalloc of *got >= bytes (a rounded size) on the current device, after giving back
// what is kept of it if that does not fit at first; of the bytes themselves (*got is set
// to them) where the rounding is what does not fit.
cudaError_t device_malloc(void** p, size_t bytes, size_t* got);

}  // namespace leo2d
