// Shared host/device utilities of the symprop_b200 library: error plumbing
// (C-ABI status codes + per-thread message), device buffers, and the packed
// symmetric-index arithmetic of the reference
// (include/detail/dense/symtensor_base.hpp:12-30, 42-76).
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "symprop.h"

namespace spb {

// ----------------------------------------------------------------- errors

struct Error : std::exception {
  int code;
  std::string msg;
  Error(int c, std::string m) : code(c), msg(std::move(m)) {}
  const char *what() const noexcept override { return msg.c_str(); }
};

void set_last_error(const std::string &msg);

[[noreturn]] inline void fail(int code, const char *fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  throw Error(code, buf);
}

inline void cuda_check(cudaError_t e, const char *what, const char *file, int line) {
  if (e != cudaSuccess) {
    // reset the runtime's last-error slot: a refused allocation (or another
    // non-sticky error) would otherwise resurface at the next launch check
    cudaGetLastError();
    int code = (e == cudaErrorMemoryAllocation) ? SYMPROP_ERR_OOM
               : (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver)
                   ? SYMPROP_ERR_NODEVICE
                   : SYMPROP_ERR_CUDA;
    fail(code, "%s failed: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
  }
}
#define SPB_CUDA(x) ::spb::cuda_check((x), #x, __FILE__, __LINE__)
#define SPB_LAUNCH_CHECK() ::spb::cuda_check(cudaGetLastError(), "kernel launch", __FILE__, __LINE__)

// value of a SYMPROP_DEBUG_* key, and whether it refuses an allocation (capi.cu)
uint64_t debug_value(int key);
bool debug_refuses(size_t bytes);

// Runs `body` and converts exceptions into a status code (C-ABI boundary).
template <class F> int guard(F &&body) {
  try {
    body();
    return SYMPROP_OK;
  } catch (const Error &e) {
    set_last_error(e.msg);
    return e.code;
  } catch (const std::bad_alloc &) {
    set_last_error("host allocation failed");
    return SYMPROP_ERR_OOM;
  } catch (const std::exception &e) {
    set_last_error(e.what());
    return SYMPROP_ERR_INVALID;
  }
}

// ------------------------------------------------------------ NVTX ranges
// Named host phases for nsys / ncu --nvtx (the GPU counterpart of the
// reference's FunctionTimer scopes, src/utils/function_timer.cpp); the calls
// do nothing unless a profiling tool is attached.
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};

// ---------------------------------------------------------- device buffer

// The library's stream-ordered memory pool of the current device (dense.cu);
// trim_pool waits for the device and gives it the unused memory back.
cudaMemPool_t device_pool();
void trim_pool();

// cudaMalloc, or with `pool` an allocation of it on st.  A refused one is tried again
// once the pool has given its unused memory back: it may hold what is missing.
inline void *device_alloc(size_t bytes, cudaMemPool_t pool = nullptr, cudaStream_t st = 0) {
  void *p = nullptr;
  auto take = [&] {
    if (debug_refuses(bytes)) return cudaErrorMemoryAllocation;
    return pool ? cudaMallocFromPoolAsync(&p, bytes, pool, st) : cudaMalloc(&p, bytes);
  };
  cudaError_t e = take();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    trim_pool();
    e = take();
  }
  SPB_CUDA(e);
  return p;
}

template <class T> struct DBuf {
  T *p = nullptr;
  size_t n = 0;
  DBuf() = default;
  explicit DBuf(size_t count) { alloc(count); }
  DBuf(const DBuf &) = delete;
  DBuf &operator=(const DBuf &) = delete;
  DBuf(DBuf &&o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }
  DBuf &operator=(DBuf &&o) noexcept {
    if (this != &o) { release(); p = o.p; n = o.n; o.p = nullptr; o.n = 0; }
    return *this;
  }
  ~DBuf() { release(); }
  void alloc(size_t count) {
    release();
    if (count == 0) return;
    p = static_cast<T *>(device_alloc(count * sizeof(T)));
    n = count;
  }
  // grows (never shrinks); contents are not preserved
  void ensure(size_t count) {
    if (count > n) alloc(count);
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  size_t bytes() const { return n * sizeof(T); }
};

// Workspace of one call on `st` from that pool, so that a repeated call waits for
// no allocation (an FP32 Gram of 50,000 x 2,002: 1.8 to 11.8 ms with cudaMalloc
// and cudaFree per call).  Larger ones than kPoolMax are not kept: they are
// allocated and freed by themselves.
struct PoolBuf {
  static constexpr size_t kPoolMax = 9ull << 29;  // 4.5 GB
  void *p = nullptr;
  cudaStream_t st;
  bool pooled = true;
  PoolBuf(size_t bytes, cudaStream_t s, size_t most = kPoolMax) : st(s), pooled(bytes <= most) {
    if (bytes) p = device_alloc(bytes, pooled ? device_pool() : nullptr, st);
  }
  PoolBuf(const PoolBuf &) = delete;
  PoolBuf &operator=(const PoolBuf &) = delete;
  ~PoolBuf() {
    if (p && pooled) cudaFreeAsync(p, st);
    else if (p) cudaFree(p);
  }
  template <class T> T *as() const { return reinterpret_cast<T *>(p); }
};

// What a tensor keeps after its first call, several arrays in one allocation: of the pool
// up to kPoolMax, where it takes a few us (cudaMalloc takes 0.4 ms from 1 MB on).  Freed
// when the device is done with it, on whichever stream.
struct KeptBuf {
  static constexpr size_t kPoolMax = size_t(64) << 20;
  char *p = nullptr;
  int dev = 0;
  bool pooled = false;
  KeptBuf() = default;
  KeptBuf(const KeptBuf &) = delete;
  KeptBuf &operator=(const KeptBuf &) = delete;
  void alloc(size_t bytes, cudaStream_t st) {
    if (!bytes) return;
    SPB_CUDA(cudaGetDevice(&dev));
    pooled = bytes <= kPoolMax;
    p = static_cast<char *>(device_alloc(bytes, pooled ? device_pool() : nullptr, st));
  }
  ~KeptBuf() {
    if (!p) return;
    int cur = dev;
    cudaGetDevice(&cur);
    if (cur != dev) cudaSetDevice(dev);
    if (pooled) cudaDeviceSynchronize();  // cudaFree does not wait for memory of a pool
    cudaFree(p);
    if (cur != dev) cudaSetDevice(cur);
  }
};

// Places of arrays that share one allocation, each on 256 bytes.
struct Places {
  size_t bytes = 0;
  template <class T> size_t add(size_t count) {
    const size_t at = bytes;
    bytes += (count * sizeof(T) + 255) / 256 * 256;
    return at;
  }
};

// ------------------------------------------------------- packed indexing

inline uint64_t binom(uint64_t n, uint64_t k) {
  if (k > n) return 0;
  if (2 * k > n) k = n - k;
  if (k == 0) return 1;
  uint64_t r = n;
  for (uint64_t i = 2; i <= k; ++i) {
    r *= (n - i + 1);
    r /= i;
  }
  return r;
}
// number of sorted order-`order` multi-indices over [0, dim)
inline uint64_t symsize(uint64_t dim, uint64_t order) { return binom(order + dim - 1, order); }

__host__ __device__ inline uint64_t factorial_u64(int k) {
  uint64_t f = 1;
  for (int i = 2; i <= k; ++i) f *= (uint64_t)i;
  return f;
}

// Host enumeration of sorted multi-indices of length `order` over [0,dim) in
// the reference's lexicographic packed order.  Calls f(idx, linear).
template <class F> void for_each_sorted(uint32_t dim, int order, F &&f) {
  std::vector<uint32_t> q((size_t)order, 0);
  uint64_t lin = 0;
  if (dim == 0) return;
  if (order == 0) { f(q, lin); return; }
  while (true) {
    f(q, lin);
    ++lin;
    int j = order - 1;
    while (j >= 0 && q[(size_t)j] + 1 >= dim) --j;
    if (j < 0) break;
    q[(size_t)j]++;
    for (int k = j + 1; k < order; ++k) q[(size_t)k] = q[(size_t)j];
  }
}

inline int bits_for(uint64_t v) {  // bits to hold values in [0, v]
  int b = 1;
  while ((v >> b) != 0) ++b;
  return b;
}

}  // namespace spb
