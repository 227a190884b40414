// common.cuh -- shared infrastructure of the GB300 engine: status handling,
// device allocation bookkeeping, exact (non-contracted) complex arithmetic.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/qudrip_gb300.h"

namespace qd {

// ---------------------------------------------------------------- errors
void set_error(const char* fmt, ...);
void clear_error();

struct Error {
  qd_status code;
};

#define QD_CUDA(call)                                                                  \
  do {                                                                                 \
    cudaError_t e__ = (call);                                                          \
    if (e__ != cudaSuccess) {                                                          \
      ::qd::set_error("%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e__)); \
      throw ::qd::Error{e__ == cudaErrorMemoryAllocation ? QD_ERR_OOM : QD_ERR_CUDA};  \
    }                                                                                  \
  } while (0)

#define QD_REQUIRE(cond, code, ...)   \
  do {                                \
    if (!(cond)) {                    \
      ::qd::set_error(__VA_ARGS__);   \
      throw ::qd::Error{code};        \
    }                                 \
  } while (0)

#define QD_LAUNCHED(ctx) ((ctx)->launches++)

#define QD_CHECK_LAUNCH()                                                              \
  do {                                                                                 \
    cudaError_t e__ = cudaGetLastError();                                              \
    if (e__ != cudaSuccess) {                                                          \
      ::qd::set_error("%s:%d kernel launch: %s", __FILE__, __LINE__, cudaGetErrorString(e__)); \
      throw ::qd::Error{QD_ERR_CUDA};                                                  \
    }                                                                                  \
  } while (0)

// Wrap a C-ABI body: converts thrown qd::Error into a status code.
template <typename F>
qd_status guard(F&& f) {
  try {
    clear_error();
    f();
    return QD_OK;
  } catch (const Error& e) {
    return e.code;
  } catch (...) {
    set_error("unexpected host exception");
    return QD_ERR_INVALID;
  }
}

// ---------------------------------------------------------------- device buffers
// Stream on which this thread's DBuf allocations are ordered.  Null (the
// default) means cudaMalloc / cudaFree.  Request-loop worker threads set their
// lane's stream, so their allocations come from the stream-ordered pool
// (cudaMallocAsync / cudaFreeAsync), which does not serialise the other
// lanes' kernels the way cudaMalloc / cudaFree do.
inline cudaStream_t& alloc_stream() {
  static thread_local cudaStream_t s = nullptr;
  return s;
}
struct AllocStreamScope {
  cudaStream_t prev;
  explicit AllocStreamScope(cudaStream_t s) : prev(alloc_stream()) { alloc_stream() = s; }
  ~AllocStreamScope() { alloc_stream() = prev; }
};

// Freed device buffers of one context, kept for its next allocations of about
// their size.  Building an operator makes and frees some forty buffers, and
// cudaMalloc and cudaFree (which waits for the device) were a third of the
// 2.85 ms that a new 20-site operator, its sector and an energy took (2.0
// without them).  A context's work is on one stream
// (a side stream joins it before its buffers are freed), so a buffer taken
// again is used after everything that used it before.  States are not taken
// from here: their addresses are handed out, and a caller may read them on a
// stream of its own until they are freed.  At most kDevCacheBytes are kept
// (larger buffers never); everything is given back with the context, and every
// context's when an allocation of any of them, or of a server's pool, fails.
constexpr size_t kDevCacheBytes = (size_t)1 << 30;
constexpr size_t kDevCacheBlock = (size_t)1 << 28;
struct DevCache {
  std::mutex lock;  // handles may be dropped on another thread than the one that works
  std::multimap<size_t, void*> idle;
  size_t held = 0;
  bool closed = false;
  // Buffers of one size class take each other's place: eighths of a power of
  // two, 512 bytes at least; what is too large to be kept is not rounded.
  static size_t round_up(size_t bytes) {
    if (bytes > kDevCacheBlock) return bytes;
    size_t step = 512;
    while (step * 16 <= bytes) step *= 2;
    return (bytes + step - 1) / step * step;
  }
  void* take(size_t bytes) {
    std::lock_guard<std::mutex> g(lock);
    auto it = idle.find(bytes);
    if (it == idle.end()) return nullptr;
    void* p = it->second;
    idle.erase(it);
    held -= bytes;
    return p;
  }
  bool give(void* p, size_t bytes) {
    std::lock_guard<std::mutex> g(lock);
    if (closed || bytes > kDevCacheBlock || held + bytes > kDevCacheBytes) return false;
    idle.emplace(bytes, p);
    held += bytes;
    return true;
  }
  void drain(bool close = false) {
    std::lock_guard<std::mutex> g(lock);
    for (auto& e : idle) cudaFree(e.second);
    idle.clear();
    held = 0;
    closed |= close;
  }
  ~DevCache() { drain(true); }
};
// The caches of all contexts: what one keeps may be what another misses.  (Never destroyed, so that contexts
// may go at any time.)
struct DevCaches {
  std::mutex lock;
  std::vector<std::weak_ptr<DevCache>> all;
  static DevCaches& get() {
    static DevCaches* c = new DevCaches;
    return *c;
  }
  std::shared_ptr<DevCache> make() {
    auto c = std::make_shared<DevCache>();
    std::lock_guard<std::mutex> g(lock);
    size_t k = 0;
    for (auto& w : all)
      if (!w.expired()) all[k++] = w;
    all.resize(k);
    all.push_back(c);
    return c;
  }
  void drain() {
    std::vector<std::shared_ptr<DevCache>> live;
    {
      std::lock_guard<std::mutex> g(lock);
      for (auto& w : all)
        if (auto c = w.lock()) live.push_back(std::move(c));
    }
    for (auto& c : live) c->drain();
  }
};
// The cache that this thread's DBuf allocations come from; null: plain cudaMalloc.
inline std::shared_ptr<DevCache>& alloc_cache() {
  static thread_local std::shared_ptr<DevCache> c;
  return c;
}
struct AllocCacheScope {
  std::shared_ptr<DevCache> prev;
  explicit AllocCacheScope(const std::shared_ptr<DevCache>& c) : prev(alloc_cache()) { alloc_cache() = c; }
  ~AllocCacheScope() { alloc_cache() = std::move(prev); }
};

// Owning device buffer; never copied.
template <typename T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  cudaStream_t s = nullptr;  // stream the buffer was allocated on (stream-ordered pool), or null
  std::shared_ptr<DevCache> c;  // the cache it goes back to, or null
  DBuf() = default;
  explicit DBuf(size_t count) { alloc(count); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n), s(o.s), c(std::move(o.c)) {
    o.p = nullptr;
    o.n = 0;
    o.s = nullptr;
  }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      n = o.n;
      s = o.s;
      c = std::move(o.c);
      o.p = nullptr;
      o.n = 0;
      o.s = nullptr;
    }
    return *this;
  }
  ~DBuf() { release(); }
  void alloc(size_t count) {
    release();
    if (count == 0) count = 1;
    s = alloc_stream();
    size_t b = count * sizeof(T);
    if (!s && alloc_cache()) {
      c = alloc_cache();
      b = DevCache::round_up(b);
      p = static_cast<T*>(c->take(b));
    }
    auto get = [&] { return s ? cudaMallocAsync((void**)&p, b, s) : cudaMalloc((void**)&p, b); };
    if (!p && get() != cudaSuccess) {
      cudaGetLastError();
      DevCaches::get().drain();
      const cudaError_t e = get();
      if (e != cudaSuccess) {
        p = nullptr;
        c.reset();
        QD_CUDA(e);
      }
    }
    n = count;
  }
  void release() {
    if (p) {
      if (s)
        cudaFreeAsync(p, s);
      else if (!c || !c->give(p, DevCache::round_up(n * sizeof(T))))
        cudaFree(p);
    }
    p = nullptr;
    n = 0;
    s = nullptr;
    c.reset();
  }
  size_t bytes() const { return n * sizeof(T); }
};

// ---------------------------------------------------------------- context
struct Ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 0;
  int64_t launches = 0;
  cudaEvent_t events[16] = {};
  std::shared_ptr<DevCache> cache = DevCaches::get().make();
};

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

// The context's device, and its cache for the buffers that the call makes.
struct CacheGuard {
  DeviceGuard dev;
  AllocCacheScope cache;
  explicit CacheGuard(Ctx* ctx) : dev(ctx->device), cache(ctx->cache) {}
};

// Allows a kernel all the dynamic shared memory a block may have.  The limit belongs to the function, not to
// the launch: set to each launch's own size, a thread with a small one would fail another thread's larger one.
template <typename K>
inline void allow_dynamic_smem(K kern, int device) {
  cudaFuncAttributes a;
  int most = 0;
  QD_CUDA(cudaFuncGetAttributes(&a, kern));
  QD_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
  QD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes));
}

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace qd

// ---------------------------------------------------------------- device math
// Complex arithmetic with one rounding per product and per sum (the
// __d*_rn intrinsics are never contracted into FMA).  This reproduces the
// reference's std::complex<double> results bit for bit.
struct __align__(16) cplx {
  double re, im;
};

__host__ __device__ inline cplx mkc(double r, double i) {
  cplx c;
  c.re = r;
  c.im = i;
  return c;
}

#ifdef __CUDACC__
__device__ __forceinline__ cplx cmul_rn(cplx a, cplx b) {
  return mkc(__dsub_rn(__dmul_rn(a.re, b.re), __dmul_rn(a.im, b.im)),
             __dadd_rn(__dmul_rn(a.re, b.im), __dmul_rn(a.im, b.re)));
}
__device__ __forceinline__ cplx cadd_rn(cplx a, cplx b) {
  return mkc(__dadd_rn(a.re, b.re), __dadd_rn(a.im, b.im));
}
__device__ __forceinline__ cplx rmul_rn(double r, cplx b) {
  return mkc(__dmul_rn(r, b.re), __dmul_rn(r, b.im));
}
#endif
