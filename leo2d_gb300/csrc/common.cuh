// common.cuh - context, errors, device buffers and launch helpers shared by
// every translation unit of libleo2d_gb300.so.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <set>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "mem_pool.h"

#include "../../include/leo2d_gpu.h"

namespace leo2d {

struct Error : std::exception {
  leo2d_status status;
  std::string msg;
  Error(leo2d_status s, std::string m) : status(s), msg(std::move(m)) {}
  const char* what() const noexcept override { return msg.c_str(); }
};

[[noreturn]] inline void fail(leo2d_status s, const std::string& m) { throw Error(s, m); }

#define LEO_CUDA(call)                                                                  \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) {                                                            \
      if (e_ == cudaErrorMemoryAllocation)                                              \
        ::leo2d::fail(LEO2D_ERR_OOM, std::string(#call) + ": " + cudaGetErrorString(e_)); \
      ::leo2d::fail(LEO2D_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));  \
    }                                                                                   \
  } while (0)

#define LEO_REQUIRE(cond, msg)                          \
  do {                                                  \
    if (!(cond)) ::leo2d::fail(LEO2D_ERR_BAD_ARG, msg); \
  } while (0)

// Largest single device allocation the calling context allows, in bytes (0: no
// limit): the context's "alloc_cap_mb" option, in force for the duration of one
// API call (guard() sets it for the calling thread).
inline thread_local size_t g_alloc_cap = 0;

// The size an allocation is rounded up to, so that jobs of nearly equal sizes find
// each other's blocks: whole driver pages from 1 MB on, steps of a sixteenth above
// 32 MB and of 64 MB from 1 GB on.
inline size_t pool_size(size_t bytes) {
  size_t unit = 512;
  if (bytes >= ((size_t)1 << 20))
    for (unit = (size_t)2 << 20; unit < ((size_t)64 << 20) && unit * 32 <= bytes;) unit *= 2;
  return (bytes + unit - 1) / unit * unit;
}

// The pool of the context whose call runs on this thread (guard() sets it).
inline thread_local const std::shared_ptr<MemPool>* g_pool = nullptr;

// Free and total memory of the current device, counting what its pools keep as free.
void device_mem_info(size_t* free_bytes, size_t* total_bytes);

// Owning device allocation (move-only).
template <class T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  DevBuf() = default;
  explicit DevBuf(size_t count) { alloc(count); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept { take_from(o); }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      take_from(o);
    }
    return *this;
  }
  ~DevBuf() { release(); }
  void alloc(size_t count) {
    release();
    if (count == 0) return;
    if (g_alloc_cap && count * sizeof(T) > g_alloc_cap)
      fail(LEO2D_ERR_OOM, "device allocation of " + std::to_string(count * sizeof(T)) +
                              " bytes exceeds the context's alloc_cap_mb");
    size_t got = pool_size(count * sizeof(T));
    void* q = g_pool ? (*g_pool)->take(got, &got) : nullptr;
    if (!q) LEO_CUDA(device_malloc(&q, count * sizeof(T), &got));
    if (g_pool) home_ = *g_pool;
    p = static_cast<T*>(q);
    held_ = got;
    n = count;
  }
  void release() {
    if (p && !(home_ && (!g_pool || *g_pool == home_) && home_->give(p, held_))) cudaFree(p);
    home_.reset();
    p = nullptr;
    n = held_ = 0;
  }
  size_t bytes() const { return n * sizeof(T); }

 private:
  void take_from(DevBuf& o) noexcept {
    p = o.p;
    n = o.n;
    held_ = o.held_;
    home_ = std::move(o.home_);
    o.p = nullptr;
    o.n = o.held_ = 0;
  }
  size_t held_ = 0;                // bytes behind p
  std::shared_ptr<MemPool> home_;  // the pool it returns to
};

struct KStat {
  int64_t launches = 0;
  double ms = 0.0;
};

struct PendingTimer {
  std::string name;
  cudaEvent_t start, stop;
};

constexpr int kTileStages = 2, kTileChunk = 4;  // the tiled step's defaults

// Device-side status word written by bounded waits (see kStatus*).
enum : int { kStatusOk = 0, kStatusTimeout = 1, kStatusNonfinite = 2, kStatusBadIndex = 3 };

}  // namespace leo2d

struct leo2d_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string last_error;
  uint64_t spin_limit = 1ull << 26;
  bool profiling = false;
  int sm_count = 0;
  size_t l2_bytes = 0;
  size_t smem_optin = 0;
  std::map<std::string, leo2d::KStat> stats;
  std::vector<leo2d::PendingTimer> pending;
  std::vector<cudaEvent_t> free_events;
  int64_t launches = 0;
  int kernel_variant = -1;    // -1 autotuned, 0 tiled gathers, 1 register gathers, 2 tensor cores, 3 row blocks,
                              // 5 row blocks of 8 on the tensor cores
  int rb_packed = -1;         // row-block step: paired FP32 FMAs (fma.rn.f32x2): -1 autotuned, 0 no, 1 yes
  int rb_warps = 0;           // row-block step: warps per block (= row blocks per tile): 0 autotuned, 16, 24, 32
  int rb_unroll = 0;          // row-block step: slot batches in flight per lane: 0 autotuned, 4, 8
  int rb_window = -1;         // row-block step over shared-memory windows: -1 autotuned, 0 no, 1 yes
  int rt_warps = 0;           // 8-row tensor-core step: warps per CTA: 0 autotuned, 8, 12, 16, 24
  int rt_depth = 0;           // 8-row tensor-core step: k-steps of T_n rows in flight per warp: 0 autotuned,
                              // 2, 3, 4, 6 (rows in registers) or 3, 7 (shared memory)
  int rt_stage = -1;          // 8-row tensor-core step: T_n rows staged in -1 autotuned, 0 registers, 1 shared memory
                              // by cp.async, 2 shared memory by TMA gathers
  int rt_rows = 0;            // tensor-core row-block step: rows per block: 0 autotuned, 8, 16
  int rt_group = 0;           // 8-row tensor-core step: consecutive blocks per warp run: 0 default (2), 1..16
  int rt_chunk = 0;           // 8-row tensor-core step: tiles per CTA between grid-wide jumps: 0 default (2)
  int reorder_curve = 1;      // locality ordering inside a patch: 1 sheet then a fine Hilbert curve, 0 reference index
  int tile_stages = leo2d::kTileStages;  // shared-memory stages of the tiled kernel
  int test_unsatisfied_wait = 0;  // test hook: tiled steps first wait on a barrier nobody completes
  bool tc_gemm_ready = false;     // shared-memory attributes of the tensor-core GEMM set on this device
  int tile_chunk = leo2d::kTileChunk;    // consecutive tiles per block between grid-wide jumps
  int tile_warps = 0;         // warps per block of the tiled kernel (0 = per shape, 8 or 24)
  int reorder = -1;           // locality ordering: -1 auto, 0 off, 1 on
  double reorder_patch = 0.0;   // patch edge (A); 0: the step kernel's own (16 A; 32 A for row blocks)
  size_t alloc_cap = 0;       // largest single device allocation of a call, bytes (0: no limit)
  int kubo_velocity = -1;     // Kubo trace: -1 D built in the row-block step where possible, 0 stored dxH
  int64_t kubo_chunk = 0;     // Kubo trace: B-side moments held at once (0: as many as memory allows)
  int mlp_fused = 1;          // network forward over many sites: 1 one fused launch, 0 one GEMM per layer
  std::shared_ptr<leo2d::MemPool> pool;   // released device memory kept for the next allocations
  std::set<const void*> smem_ready;       // kernels allowed the device's largest dynamic shared memory
  leo2d::DevBuf<int> status;  // one int, reset before kernels that may set it
  leo2d::DevBuf<char> scratch;  // small work arrays of the transforms (ctx_scratch)
};

namespace leo2d {

// Runs f, converting exceptions into a status and the context's last error.
template <class F>
leo2d_status guard(leo2d_ctx* ctx, F&& f) {
  struct CapScope {  // the context's allocation cap for this call, restored on exit
    size_t saved;
    explicit CapScope(size_t cap) : saved(g_alloc_cap) { g_alloc_cap = cap; }
    ~CapScope() { g_alloc_cap = saved; }
  } cap_scope(ctx ? ctx->alloc_cap : g_alloc_cap);
  struct PoolScope {
    const std::shared_ptr<MemPool>* saved;
    explicit PoolScope(const std::shared_ptr<MemPool>* p) : saved(g_pool) {
      g_pool = p;
      if (p) (*p)->enter();
    }
    ~PoolScope() {
      if (g_pool) (*g_pool)->leave();
      g_pool = saved;
    }
  } pool_scope(ctx && ctx->pool ? &ctx->pool : g_pool);
  // a call that fails leaves nothing running on memory that its buffers gave back
  struct Drain {
    leo2d_ctx* ctx;
    bool armed = true;
    ~Drain() {
      if (armed && ctx && ctx->stream) cudaStreamSynchronize(ctx->stream);
    }
  } drain{ctx};
  try {
    f();
    drain.armed = false;
    if (ctx) ctx->last_error.clear();
    return LEO2D_OK;
  } catch (const Error& e) {
    if (ctx) ctx->last_error = e.msg;
    return e.status;
  } catch (const std::bad_alloc&) {
    if (ctx) ctx->last_error = "host allocation failed";
    return LEO2D_ERR_OOM;
  } catch (const std::exception& e) {
    if (ctx) ctx->last_error = e.what();
    return LEO2D_ERR_CUDA;
  } catch (...) {
    if (ctx) ctx->last_error = "unknown error";
    return LEO2D_ERR_CUDA;
  }
}

// Lets `kern` be launched with any dynamic shared memory the device has, once per
// context. The limit belongs to the function on the device, not to a context: a call
// that sets it to one launch's size can undercut another thread between its own call
// and its launch, so it is set nowhere else. (Setting it before every launch also
// cost a Chebyshev step of a small cell 1.2 us of its 7.)
inline void allow_smem(leo2d_ctx* ctx, const void* kern) {
  if (ctx->smem_ready.count(kern)) return;
  cudaFuncAttributes at{};
  LEO_CUDA(cudaFuncGetAttributes(&at, kern));
  LEO_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(ctx->smem_optin - at.sharedSizeBytes)));
  ctx->smem_ready.insert(kern);
}

cudaEvent_t ctx_event(leo2d_ctx* ctx);
// Synchronises the context stream and folds finished timers into the stats.
void ctx_sync(leo2d_ctx* ctx);
// Reads and clears the device status word; throws on a non-zero code.
void ctx_check_status(leo2d_ctx* ctx, const char* where);

// Launches `f` (which enqueues exactly one kernel on ctx->stream), counts it and,
// when profiling is on, brackets it with CUDA events on the same stream.
template <class F>
void launch(leo2d_ctx* ctx, const char* name, F&& f) {
  cudaEvent_t a = nullptr, b = nullptr;
  if (ctx->profiling) {
    a = ctx_event(ctx);
    b = ctx_event(ctx);
    LEO_CUDA(cudaEventRecord(a, ctx->stream));
  }
  f();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) fail(LEO2D_ERR_CUDA, std::string("launch of ") + name + ": " + cudaGetErrorString(e));
  ctx->launches += 1;
  if (ctx->profiling) {
    LEO_CUDA(cudaEventRecord(b, ctx->stream));
    ctx->pending.push_back(PendingTimer{name, a, b});
  } else {
    ctx->stats[name].launches += 1;
  }
}

inline unsigned grid_for(int64_t work, int per_block, int64_t cap = (1ll << 31) - 1) {
  int64_t g = (work + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (unsigned)g;
}

template <class T>
void h2d(leo2d_ctx* ctx, T* dst, const T* src, size_t count) {
  if (count) LEO_CUDA(cudaMemcpyAsync(dst, src, count * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
}
template <class T>
void d2h(leo2d_ctx* ctx, T* dst, const T* src, size_t count) {
  if (count) LEO_CUDA(cudaMemcpyAsync(dst, src, count * sizeof(T), cudaMemcpyDeviceToHost, ctx->stream));
}

// Work space of one call on this context, one live request at a time, kept up to 64 MiB (a call synchronises
// before it returns, and a context serves one thread at a time, so the next call
// may reuse it): the transforms' four allocations took longer than their kernels.
constexpr size_t kScratchKept = (size_t)64 << 20;
template <class T>
T* ctx_scratch(leo2d_ctx* ctx, size_t count) {
  const size_t bytes = count * sizeof(T);
  if (g_alloc_cap && bytes > g_alloc_cap)  // also when a kept buffer would do
    fail(LEO2D_ERR_OOM, "device allocation of " + std::to_string(bytes) + " bytes exceeds the context's alloc_cap_mb");
  if (ctx->scratch.n < bytes || (ctx->scratch.n > kScratchKept && bytes <= kScratchKept)) {
    ctx->scratch.release();
    ctx->scratch.alloc(std::max(bytes, (size_t)1 << 16));
  }
  return reinterpret_cast<T*>(ctx->scratch.p);
}

// Work space of one call in several parts: together in the context's scratch or, where
// that would pass the context's limit on one allocation, an allocation each.
class Scratch {
 public:
  Scratch(leo2d_ctx* ctx, std::initializer_list<size_t> bytes) {
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    size_t total = 0;
    for (size_t b : bytes) total += up(b);
    const bool apart = g_alloc_cap && total > g_alloc_cap;
    char* p = apart ? nullptr : ctx_scratch<char>(ctx, total);
    for (size_t b : bytes) {
      if (n_ == kParts) fail(LEO2D_ERR_BAD_ARG, "too many parts of a work space");
      if (apart) {
        own_[n_].alloc(b);
        part_[n_] = own_[n_].p;
      } else {
        part_[n_] = p;
        p += up(b);
      }
      ++n_;
    }
  }
  template <class T>
  T* get(int i) const {
    return reinterpret_cast<T*>(part_[i]);
  }

 private:
  static constexpr int kParts = 5;
  int n_ = 0;
  DevBuf<char> own_[kParts];
  char* part_[kParts] = {};
};

// tab[m] = cos(pi m / (2P)), 0 <= m < 4P (transform.cu).
void cos_table(leo2d_ctx* ctx, int P, double* tab);

// Exclusive prefix sum of n int64 values: out[0..n] with out[n] = total.
// `out` may alias `in` only if it is a distinct buffer of n+1 elements.
void exclusive_scan_i64(leo2d_ctx* ctx, const int64_t* in, int64_t* out, int64_t n);

// Sum of n int64 values (device), returned to the host.
int64_t reduce_sum_i64(leo2d_ctx* ctx, const int64_t* in, int64_t n);

}  // namespace leo2d
