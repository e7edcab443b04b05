// Shared parts of the S3TTMc kernels that multiply on the FP64 tensor cores
// (s3ttmc_split.cu, s3ttmc_chain5.cu, s3ttmc_chain8.cu): named barriers between the building and
// the multiplying warps, the 8 x 8 x 4 product, and the walk over a CTA's
// work items.
#pragma once

#include "check.cuh"
#include "tensor.cuh"

namespace spb {
namespace {

template <int THREADS> __device__ __forceinline__ void bar_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}
template <int THREADS> __device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}

// c (8 x 8, rows r8 = lane / 4, columns 2 kq + {0, 1}, kq = lane % 4) +=
// a (8 x 4: row r8, column kq) * b (4 x 8: row kq, column r8)
__device__ __forceinline__ void mma_f64(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) { mma_f64(c[0], c[1], a, b); }

// (d0, d1) += (a, a) * (b0, b1) in one paired FP32 FMA: each half rounds as a
// scalar fmaf does
__device__ __forceinline__ void fma2(float &d0, float &d1, float a, float b0, float b1) {
  unsigned long long d, x, y;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(d0), "f"(d1));
  asm("mov.b64 %0, {%1, %1};" : "=l"(x) : "f"(a));
  asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b0), "f"(b1));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(x), "l"(y));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d0), "=f"(d1) : "l"(d));
}

// A CTA's stages in order: the entries [ob, oe) of items blockIdx.x,
// blockIdx.x + gridDim.x, ..., K at a time.  Both roles walk the same sequence.
// P has chunks, nchunks, nentries (the bound of ob, oe), nrows and nslots.
template <int K> struct Walk {
  uint32_t item = 0, row = 0, slot = 0, o = 0, oe = 0;
  bool first = false;  // the item's first stage
  Chunk ahead{};       // the item to be opened next, loaded an item early
  template <class P> __device__ __forceinline__ void start(const P &p) {
    item = blockIdx.x;
    if (item < p.nchunks) ahead = p.chunks[item];
  }
  template <class P> __device__ __forceinline__ bool valid(const P &p) const { return item < p.nchunks; }
  __device__ __forceinline__ int count() const { return (int)min((uint32_t)K, oe - o); }
  __device__ __forceinline__ bool last() const { return oe - o <= (uint32_t)K; }
  // opens the first item with entries at or after `item`; empty(row, slot)
  // is called for each one without
  template <class P, class Empty> __device__ __forceinline__ void open(const P &p, Empty &&empty) {
    for (; item < p.nchunks; item += gridDim.x) {
      const Chunk ch = ahead;
      if (item + gridDim.x < p.nchunks) ahead = p.chunks[item + gridDim.x];
      if (!SPB_BOUND(ch.ob <= ch.oe && ch.oe <= p.nentries && ch.row < p.nrows &&
                         (ch.slot == kDirect || ch.slot < p.nslots),
                     501, item))
        continue;
      row = ch.row;
      slot = ch.slot;
      o = (uint32_t)ch.ob;
      oe = (uint32_t)ch.oe;
      first = true;
      if (o < oe) return;
      empty(row, slot);
    }
  }
  template <class P, class Empty> __device__ __forceinline__ void next(const P &p, Empty &&empty) {
    if (!last()) {
      o += K;
      first = false;
    } else {
      item += gridDim.x;
      open(p, empty);
    }
  }
};

// one entry of a finished item: of its row of Y, or of its partial row
template <typename T, class P>
__device__ __forceinline__ void put(const P &p, uint32_t row, uint32_t slot, uint32_t e, double y) {
  if (slot == kDirect) reinterpret_cast<T *>(p.Y)[(uint64_t)row * p.m + e] = (T)y;
  else p.partials[(uint64_t)slot * p.m + e] = y;
}

}  // namespace
}  // namespace spb
