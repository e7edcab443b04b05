// FP64 column Gram C = A^T A on the 8-bit integer tensor cores (tcgen05
// kind::i8): HOOI's dense step in FP64 (src/sparse/spsymtensor.cpp:225,
// src/dense/matrixops.cpp:18-43 form it with LAPACK).
//
// Method: Ozaki scheme II (Ozaki, Uchino, Imamura 2025), a matrix product of
// integers by the Chinese remainder theorem.  The rows are taken in chunks of
// at most kMaxChunk.  In a chunk every column is scaled by a power of two so
// that its largest magnitude is in [2^52, 2^53) and rounded to integers,
//     a_kj = 2^-s_j n_kj + delta,  |delta| <= 2^-s_j / 2  (exact to 2^-53 of
//     the column's largest entry of the chunk),
// and sum_k n_ki n_kj, an integer of at most 2^122, is found from its residues
// modulo 16 pairwise coprime p <= 256 (product 2^125.4): residues of the n_kj
// fit 8 bits, each modulus is one int8 product with exact int32 sums
// (at most chunk * 2^14 = 2^30), and the sum is put together in 128-bit integers and
// rounded once.  The chunks' sums are added in FP64.  No accumulation error
// grows with the number of rows: the error is that of the scaled rounding,
// 2^-54 of the column maximum per entry with random sign, and of one rounding
// per chunk.
//
// What the rounding may cost an entry.  With P_j = 2^(53 - s_j) (the power of
// two above column j's largest magnitude of a chunk) the entry (i, j) is off by at
// most 2^-54 sum_k (|a_ki| P_j + |a_kj| P_i): small against |a_i| |a_j|, which is
// all that an eigenvalue problem asks for, but not against
// T_ij = sum_k |a_ki| |a_kj|, the scale of a sum in floating point, where the
// columns' large entries lie in different rows.  A caller that wants every
// entry (componentwise) gets this checked first: |a_kj| / P_j in 7 bits, rounded
// down, gives a lower bound W of T / (P_i P_j) by one more product, and with
// N_j = |a_j| / P_j (2-norm) an entry is kept where
//     N_i + N_j <= sqrt(rows of the chunk) W      in every chunk.
// Then sum |a_ki| <= sqrt(rows) N_i P_i makes its error at most
// rows / 2 * 2^-53 T_ij, half the bound of a sum of `rows` terms in floating
// point, and (the roundings having random signs) 0.3 sqrt(rows) 2^-53 T_ij in the
// root mean square, what a floating-point sum of terms of one sign is off by.
// The other entries are summed in FP64 (pair_kernel), or all of them by the
// caller when they are many.
//
// Bound: 16 int8 products over the upper 256 x 256 tiles.  200,000 x 3,876:
// 136 tiles, 5.7e13 integer operations (12.7 ms at the nominal 4.5 POP/s),
// against 3.0e12 FP64 operations (81 ms at the nominal 37 TFLOP/s) for the
// CUDA-core kernel in dense.cu (137 ms).  Measured 27.4 ms (with the check 28.4): product 17.9 (3.2
// POP/s), residues 5.8 (reads A, writes 16 bytes per entry), remainders 1.1,
// column maxima 0.9; error against 64 bits 1.2e-16, 6.2e-15 for the CUDA-core
// kernel.  Running the residues and remainders on a second stream beside the
// product gave nothing (29.0 against 28.9 ms).
//
// Kernel (i8_gram_kernel): one CTA of 256 threads per (tile, modulus, chunk),
// 256 x 256 outputs as two M = 128, N = 256 accumulators that fill the tensor
// memory (64 KB of operands per 128-wide k block and 1024 tensor clocks: the
// 128 x 256 tile of gram_tc.cu would read 1.5 times as much of them from L2).
// Warp 0 loads (TMA, 128-byte swizzle, 3 stages), warp 1 issues, all 8 warps
// reduce the sums modulo p and store one byte per entry.  Waits are bounded
// as in gram_tc.cu.
#include <algorithm>
#include <cmath>
#include <optional>

#include "gram_i8.cuh"
#include "gram_tc.cuh"
#include "tcgen05.cuh"

namespace spb {
namespace gram {
namespace {

constexpr int kP = 16;
constexpr int kModulus[kP] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
constexpr int kMinChunk = 1024, kMaxChunk = 65536;  // rows: 2^16 * 2^106 < P / 8 and 2^16 * 2^14 = 2^30
constexpr int kTile = 256, kBK = 128, kNStages = 3;
constexpr uint32_t kOperand = kTile * kBK;  // bytes
constexpr size_t kSmem = (size_t)kNStages * 2 * kOperand + 1024;

// (P / p)^-1 mod p of every modulus, and P / p and P as two 64-bit words
struct Crt {
  uint32_t inv[kP];
  unsigned long long wlo[kP], whi[kP], plo, phi;
  double rp[kP];  // 1 / p
};

constexpr Crt make_crt() {
  Crt t{};
  unsigned __int128 P = 1;
  for (int i = 0; i < kP; ++i) P *= (unsigned)kModulus[i];
  t.plo = (unsigned long long)P;
  t.phi = (unsigned long long)(P >> 64);
  for (int i = 0; i < kP; ++i) {
    const unsigned p = (unsigned)kModulus[i];
    const unsigned __int128 w = P / p;
    t.wlo[i] = (unsigned long long)w;
    t.whi[i] = (unsigned long long)(w >> 64);
    const unsigned r = (unsigned)(w % p);
    for (unsigned x = 1; x < p; ++x)
      if (r * x % p == 1) t.inv[i] = x;
    t.rp[i] = 1.0 / p;
  }
  return t;
}
__constant__ Crt c_crt = make_crt();
__constant__ int c_mod[kP] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};

// ------------------------------------------------------------ preparation

// Bits of the largest magnitude of every column of every chunk (magnitudes
// order as integers; an infinity or a NaN comes out on top)
__global__ void __launch_bounds__(128) col_max_kernel(const double *__restrict__ A, int rows, int cols, int lda,
                                                      int chunk, int part, unsigned long long *__restrict__ cmax) {
  const int c = blockIdx.x * 128 + threadIdx.x;
  const int k0 = blockIdx.y * chunk + blockIdx.z * part, k1 = min(min(rows, (int)(blockIdx.y + 1) * chunk), k0 + part);
  if (c >= cols || k0 >= k1) return;
  unsigned long long m = 0;
#pragma unroll 8
  for (int k = k0; k < k1; ++k) m = max(m, __double_as_longlong(A[(size_t)k * lda + c]) & 0x7fffffffffffffffull);
  atomicMax(&cmax[(size_t)blockIdx.y * cols + c], m);
}

// Entries of a componentwise Gram that have to be summed in FP64.  Past the limit
// the FP64 kernel does all of them, and what is still queued returns at once.
struct Odd {
  int2 *pairs;
  unsigned *count, max;
  __device__ __forceinline__ bool too_many() const { return *(volatile unsigned *)count > max; }
};

// Exponent s of every column: |a| 2^s < 2^53; *bad is set when one is not finite
__global__ void scale_kernel(const unsigned long long *cmax, int n, int *s, int *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long b = cmax[i];
  if (b >= 0x7ff0000000000000ull) *bad = 1;
  int e = 0;
  if (b) frexp(__longlong_as_double((long long)b), &e);  // |a| < 2^e
  s[i] = b ? 53 - e : 0;
}

// Residues of the scaled columns: out[(chunk * planes + p) * cols + c][k], k < kc
// bytes contiguous (rows past the chunk's end are zero).  A thread takes 32
// rows of one column: a warp reads 256-byte row pieces, and every store fills a
// 32-byte sector.  q = round(n / p) is within 2^-7 of n / p + 1/2, so |r|
// may pass p / 2 by 2: put back into 8 bits where p / 2 + 2 > 127.
// MAG: the last plane takes |n| 2^-53 in 7 bits, rounded down, and nsq the sum of
// the squares of the same in 15 bits, rounded up (integers: the decision that
// rests on them is the same in every run); weight (or null): its sum over the columns
// for every block of 128 rows.
template <bool MAG>
__global__ void __launch_bounds__(128) residue_kernel(const double *__restrict__ A, int rows, int cols, int lda,
                                                      int chunk, int kc, const int *__restrict__ s, int chunk0,
                                                      signed char *__restrict__ out,
                                                      unsigned long long *__restrict__ nsq,
                                                      unsigned long long *__restrict__ weight, const Odd odd) {
  if (odd.too_many()) return;
  constexpr int kPlanes = kP + (MAG ? 1 : 0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  const int k0 = blockIdx.y * 128 + warp * 32;  // within the chunk
  const int ch = chunk0 + blockIdx.z;
  unsigned long long sum = 0;
  if (c < cols) {
    const int r0 = ch * chunk + k0, r1 = min(rows, (ch + 1) * chunk);
    const int sh = s[(size_t)ch * cols + c], s1 = sh / 2;
    // 2^sh as two factors: sh may lie outside the exponent range
    const double f1 = __longlong_as_double((long long)(s1 + 1023) << 52),
                 f2 = __longlong_as_double((long long)(sh - s1 + 1023) << 52);
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
    double n[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) n[i] = r0 + i < r1 ? rint(A[(size_t)(r0 + i) * lda + c] * f1 * f2) : 0.0;
    signed char *plane = out + ((size_t)blockIdx.z * kPlanes * cols + c) * kc + k0;
    auto store = [&](int p, const uint32_t (&w)[8]) {
      uint4 *o = reinterpret_cast<uint4 *>(plane + (size_t)p * cols * kc);
      o[0] = make_uint4(w[0], w[1], w[2], w[3]);
      o[1] = make_uint4(w[4], w[5], w[6], w[7]);
    };
    for (int p = 0; p < kP; ++p) {
      const double m = (double)c_mod[p], rm = c_crt.rp[p];
      uint32_t w[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint32_t v = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const double x = n[4 * q + b];
          const double t = fma(x, rm, kMagic) - kMagic;
          int r = (int)__double_as_longlong(fma(-t, m, x) + kMagic);  // the low word holds the integer
          if (p == 1 || p == 2) {  // 255, 253 (for 256 the byte wraps to the same residue)
            const int mi = c_mod[p];
            r = r > 127 ? r - mi : r < -128 ? r + mi : r;
          }
          v |= (uint32_t)(r & 0xff) << (8 * b);
        }
        w[q] = v;
      }
      store(p, w);
    }
    if constexpr (MAG) {
      uint32_t w[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        w[q] = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const float x = fabsf((float)n[4 * q + b]) * 0x1p-53f;
          w[q] |= (uint32_t)min((int)(x * 127.f), 127) << (8 * b);
          const uint32_t u = (uint32_t)ceilf(x * 32768.f);
          sum += (unsigned long long)u * u;
        }
      }
      store(kP, w);
    }
  }
  if constexpr (MAG) {
    __shared__ unsigned long long part[4][32];
    part[warp][lane] = sum;
    __syncthreads();
    if (warp == 0) {
      sum = part[0][lane] + part[1][lane] + part[2][lane] + part[3][lane];
      if (c < cols) atomicAdd(&nsq[(size_t)ch * cols + c], sum);
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0 && weight) atomicAdd(&weight[blockIdx.z * gridDim.y + blockIdx.y], sum);
    }
  }
}

// The `few` blocks of 128 rows with the largest weight, per chunk (blockIdx.x)
__global__ void __launch_bounds__(512) pick_kernel(const unsigned long long *weight, int kblocks, int few, int *picked) {
  __shared__ unsigned long long w[kMaxChunk / 128];
  const unsigned long long *mine = weight + (size_t)blockIdx.x * kblocks;
  for (int i = threadIdx.x; i < kblocks; i += 512) w[i] = mine[i];
  __syncthreads();
  for (int i = threadIdx.x; i < kblocks; i += 512) {
    int r = 0;
    for (int j = 0; j < kblocks; ++j) r += w[j] > w[i] || (w[j] == w[i] && j < i);
    if (r < few) picked[(size_t)blockIdx.x * few + r] = i;
  }
}

// The entries (i, j) of the list in FP64: C_ij = C_ji = sum_k a_ki a_kj
__global__ void __launch_bounds__(256) pair_kernel(const int2 *__restrict__ pairs, const double *__restrict__ A,
                                                   int rows, int lda, double *__restrict__ C, int ldc) {
  __shared__ double red[8];
  const int2 p = pairs[blockIdx.x];
  double sum = 0.0;
#pragma unroll 4
  for (int k = threadIdx.x; k < rows; k += 256) sum = fma(A[(size_t)k * lda + p.x], A[(size_t)k * lda + p.y], sum);
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) sum += red[w];
    C[(size_t)p.x * ldc + p.y] = sum;
    C[(size_t)p.y * ldc + p.x] = sum;
  }
}

// ---------------------------------------------------------------- product

constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTile >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t acc) {
  uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(kIdesc), "r"(acc), "r"(z), "r"(z), "r"(z), "r"(z));
}

struct I8Args {
  int cols, ntile, ntiles;    // tiles of 256 per side, upper tiles
  int kblocks;                // 128-wide blocks of a chunk
  const int *picked;          // null: all of them, else kblocks of each chunk
  unsigned char *C;           // (chunk * kP + p) planes of ld x ld residues
  int ld;
  int *err;
  uint64_t wait_ns;
  int expired_warp;           // failure injection (-1: none)
  int planes;                 // per chunk: kP of residues, one more of magnitudes
  // The first `checks` units are the products of the chunks' magnitudes: over some of the
  // rows (some: *suspect is set when an entry may have to be summed in FP64) or
  // over all (such entries go to the list; with `suspect` only when that is set).
  int checks;
  bool some;
  int *suspect;
  const unsigned long long *nsq;
  int chunk0, chunk, rows;
  Odd odd;
};

__global__ void __launch_bounds__(256, 1)
    i8_gram_kernel(const __grid_constant__ CUtensorMap map, const I8Args a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[kNStages], empty_bar[kNStages], done_bar;
  __shared__ uint32_t tmem_base_holder;
  __shared__ volatile int abort_flag;
  __shared__ volatile int progress;
  __shared__ int issued[kNStages];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // unit: tile fastest, so that the CTAs of a wave share a modulus in L2
  const int unit = (int)blockIdx.x / a.ntiles, sums = unit - a.checks;
  const bool check = sums < 0;
  const int plane = check ? unit * a.planes + kP : sums / kP * a.planes + sums % kP;
  if (a.planes > kP &&
      __syncthreads_or(threadIdx.x == 0 && (a.odd.too_many() || (check && !a.some && a.suspect && !*a.suspect))))
    return;
  int ti = 0, tj = (int)blockIdx.x - unit * a.ntiles;
  while (tj >= a.ntile - ti) {
    tj -= a.ntile - ti;
    ++ti;
  }
  tj += ti;
  const int row0 = plane * a.cols + ti * kTile, col0 = plane * a.cols + tj * kTile;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kNStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
      issued[s] = 0;
    }
    mbar_init(&done_bar, 1);
    abort_flag = 0;
    progress = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const int chunk = a.chunk0 + plane / a.planes, modulus = plane % a.planes;
  __shared__ float norm[kTile];  // check: N of the tile's columns, 0 past the last
  const unsigned long long *nsq = a.nsq + (size_t)chunk * a.cols;
  if (check) {
    const int j = tj * kTile + threadIdx.x;
    norm[threadIdx.x] = j < a.cols ? sqrtf((float)nsq[j]) * 0x1p-15f : 0.f;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_holder)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base_holder;

  if (warp == 0 && lane == 0) {
    const int *picked = a.picked ? a.picked + (size_t)(plane / a.planes) * a.kblocks : nullptr;
    for (int it = 0; it < a.kblocks; ++it) {
      const int s = it % kNStages;
      const uint32_t round = (uint32_t)(it / kNStages);
      if (it >= kNStages && !mbar_wait(&empty_bar[s], (round - 1) & 1, &abort_flag, a.wait_ns)) {
        abort_flag = 1;
        break;
      }
      unsigned char *st = smem + (size_t)s * 2 * kOperand;
      mbar_expect_tx(&full_bar[s], 2 * kOperand);
      const int x = (picked ? picked[it] : it) * kBK;
      tma_load_2d(st, &map, &full_bar[s], x, row0);
      tma_load_2d(st + kOperand, &map, &full_bar[s], x, col0);
      issued[s] = it + 1;
    }
  } else if (warp == 1 && lane == 0) {
    bool ok = true;
    for (int it = 0; it < a.kblocks; ++it) {
      const int s = it % kNStages;
      if (!mbar_wait(&full_bar[s], (uint32_t)(it / kNStages) & 1, &abort_flag, a.wait_ns)) {
        abort_flag = 1;
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t base = smem_u32(smem + (size_t)s * 2 * kOperand);
#pragma unroll
      for (int k = 0; k < kBK / 32; ++k) {  // K-major rows of 128 bytes, 32 bytes a step
        const uint64_t db = smem_desc(base + kOperand + k * 32, 16u);
        umma_i8(tmem, smem_desc(base + k * 32, 16u), db, (it > 0 || k > 0) ? 1u : 0u);
        umma_i8(tmem + 256u, smem_desc(base + 128 * kBK + k * 32, 16u), db, (it > 0 || k > 0) ? 1u : 0u);
      }
      umma_commit(&empty_bar[s]);
      progress = it + 1;
    }
    umma_commit(&done_bar);
    if (!ok) abort_flag = 1;
  }
  __syncwarp();
  const bool done = mbar_wait_progress(&done_bar, &progress) && warp != a.expired_warp;
  asm volatile("tcgen05.fence::after_thread_sync;");
  const int go = __all_sync(0xffffffffu, done ? 1 : 0) && !__shfl_sync(0xffffffffu, (int)abort_flag, 0);
  if (go && check) {
    const int half = warp >> 2, i = ti * kTile + half * 128 + (warp & 3) * 32 + lane;
    const float ni = i < a.cols ? sqrtf((float)nsq[i]) * 0x1p-15f : 0.f;
    const float unit = sqrtf((float)min(a.chunk, a.rows - chunk * a.chunk)) / (127.f * 127.f);
#pragma unroll 1
    for (int c = 0; c < kTile; c += 32) {
      uint32_t v[32];
      tmem_load<32>(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * 256 + c), v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        const float nj = norm[c + q];
        const int j = tj * kTile + c + q;
        if (ni > 0.f && nj > 0.f && i <= j && !(ni + nj <= unit * (float)(int)v[q])) {
          if (a.some) {
            *a.suspect = 1;
            continue;
          }
          // past the limit the count no longer matters (and may not wrap)
          if (a.odd.too_many()) continue;
          const unsigned at = atomicAdd(a.odd.count, 1u);
          if (at < a.odd.max) a.odd.pairs[at] = make_int2(i, j);
        }
      }
    }
  } else if (go) {
    // warp w: lanes of quadrant w % 4 of accumulator w / 4.  The sums (at most
    // 2^30 in magnitude) modulo p, times (P / p)^-1 modulo p.
    const int half = warp >> 2, r = ti * kTile + half * 128 + (warp & 3) * 32 + lane;
    const uint32_t p = (uint32_t)c_mod[modulus], inv = c_crt.inv[modulus];
    const uint32_t magic = 0xffffffffu / p, bias = (1u << 30) / p * p + p;
    unsigned char *C = a.C + (size_t)(plane / a.planes * kP + modulus) * a.ld * a.ld + (size_t)r * a.ld + tj * kTile;
#pragma unroll 1
    for (int c = 0; c < kTile; c += 32) {
      uint32_t v[32];
      tmem_load<32>(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * 256 + c), v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      uint32_t o[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        o[q] = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          uint32_t u = v[4 * q + b] + bias;  // the sum plus a multiple of p, positive
          u -= __umulhi(u, magic) * p;       // below 2 p + small: at most two subtractions
          u = u >= p ? u - p : u;
          u = u >= p ? u - p : u;
          u *= inv;
          u -= __umulhi(u, magic) * p;
          u = u >= p ? u - p : u;
          u = u >= p ? u - p : u;
          o[q] |= u << (8 * b);
        }
      }
      uint4 *d = reinterpret_cast<uint4 *>(C + c);  // rows up to ld are stored: ld is a multiple of 256
      d[0] = make_uint4(o[0], o[1], o[2], o[3]);
      d[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
  } else if (lane == 0) {  // every warp decides by its own clock
    atomicExch(a.err, 1);
  }
  if (threadIdx.x == 0 && (abort_flag || !done)) {
    for (int s = 0; s < kNStages; ++s)
      if (issued[s] > 0) {
        volatile int never = 0;
        mbar_wait(&full_bar[s], (uint32_t)((issued[s] - 1) / kNStages) & 1, &never, kWaitNs);
      }
    if (!done) {
      volatile int never = 0;
      mbar_wait(&done_bar, 0, &never, kWaitNs);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ------------------------------------------------------------- remainders

// One 32 x 32 tile (i0 <= j0) of C and its mirror image: every chunk's sum
// X = sum_p c_p (P / p) - P round(sum_p c_p / p) in 128 bits (|X| < P / 8, so the
// rounding is never in doubt), scaled back and added in FP64, chunks in order.
__global__ void __launch_bounds__(256) crt_kernel(const unsigned char *__restrict__ R, int ld, int cols, int nchunk,
                                                  int chunk0, const int *__restrict__ s, int add,
                                                  double *__restrict__ C, int ldc, const Odd odd) {
  if (blockIdx.x < blockIdx.y || odd.too_many()) return;
  __shared__ double t[32][33];
  const int j0 = blockIdx.x * 32, i0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const size_t pl = (size_t)ld * ld;
#pragma unroll 1
  for (int y = ty; y < 32; y += 8) {
    const int i = i0 + y, j = j0 + tx;
    double sum = 0.0;
    if (i < cols && j < cols) {
      if (add) sum = C[(size_t)i * ldc + j];
      for (int c = 0; c < nchunk; ++c) {
        const unsigned char *r = R + (size_t)c * kP * pl + (size_t)i * ld + j;
        unsigned long long lo = 0, hi = 0;
        double q = 0.0;
#pragma unroll
        for (int p = 0; p < kP; ++p) {
          const unsigned long long v = r[p * pl], x = v * c_crt.wlo[p];
          lo += x;
          hi += v * c_crt.whi[p] + __umul64hi(v, c_crt.wlo[p]) + (lo < x ? 1ull : 0ull);
          q += (double)v * c_crt.rp[p];
        }
        const unsigned long long k = (unsigned long long)rint(q), x = k * c_crt.plo;
        hi -= k * c_crt.phi + __umul64hi(k, c_crt.plo) + (lo < x ? 1ull : 0ull);
        lo -= x;
        const bool neg = (long long)hi < 0;
        if (neg) {
          lo = ~lo + 1;
          hi = ~hi + (lo == 0 ? 1ull : 0ull);
        }
        // hi < 2^60: bring the value to 64 bits plus a sticky bit, so that one
        // conversion rounds it
        int sh = 0;
        if (hi) {
          sh = 64 - __clzll((long long)hi);
          const unsigned long long rest = lo << (64 - sh);
          lo = (sh < 64 ? (hi << (64 - sh)) | (lo >> sh) : hi) | (rest ? 1ull : 0ull);
        }
        const double d = (double)lo;
        sum += scalbn(neg ? -d : d, sh - s[(size_t)(chunk0 + c) * cols + i] - s[(size_t)(chunk0 + c) * cols + j]);
      }
      if (i <= j) C[(size_t)i * ldc + j] = sum;
    }
    t[y][tx] = sum;
  }
  __syncthreads();
  for (int y = ty; y < 32; y += 8) {  // the mirror image: row j0 + y, column i0 + tx
    const int j = j0 + y, i = i0 + tx;
    if (i < j && j < cols) C[(size_t)j * ldc + i] = t[tx][y];
  }
}

int sms() {
  int dev = 0, n = 0;
  SPB_CUDA(cudaGetDevice(&dev));
  SPB_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
  return std::max(n, 1);
}

// Chunks of the rows.  A product takes 1024 clocks per 128 rows and about
// 12,000 besides (loads of the first stages, reduction, tensor memory), one
// per SM at a time; the remainders of a chunk are put together in 18 us at 320 columns
// (latency) and 75 us at 2,002: of the chunk counts whose operands, chunk by chunk, take at
// most `limit` bytes, the one whose waves take least.  `nchunk` is 0 when there is
// none.
// The check of a componentwise Gram is a 17th plane among the sums, or (some rows give
// a lower bound of W as well) launches before them: the eighth of the blocks of 128
// rows that holds the largest rows, and all only where that is not enough.  The second
// costs three launches, the first often a wave: 20,000 x 2,002 1.15 / 1.09 ms (without a
// check 1.03); 20,000 x 320 0.315 / 0.333, 1,536 x 715 0.150 / 0.182.  Largest rows:
// on rows with scales of a power law every 8th block left entries in doubt
// (200,000 x 3,876: 29.6 ms).
struct I8Plan {
  int ntile, ntiles, ld;
  int chunk, nchunk = 0;    // rows per chunk
  int kc, group;            // padded rows, chunks per launch
  int few = 0;              // not 0: the check by itself, over so many blocks of 128 rows first
  size_t res, bytes;        // of a launch's residues, and of all its operands
};

I8Plan plan_i8(int rows, int cols, int planes, size_t limit) {
  I8Plan g;
  g.ntile = (cols + kTile - 1) / kTile;
  g.ntiles = g.ntile * (g.ntile + 1) / 2;
  g.ld = g.ntile * kTile;
  auto res = [&](int kc, int group) { return ((size_t)group * planes * cols * kc + 255) / 256 * 256; };
  auto bytes = [&](int kc, int group) { return res(kc, group) + (size_t)group * kP * g.ld * g.ld; };
  const int n = sms();
  // the most rows of one chunk
  int most = 0;
  if (bytes(kBK, 1) <= limit) {
    most = (int)std::min<size_t>(kMaxChunk, (limit - bytes(0, 1)) / ((size_t)planes * cols));
    most = most / kBK * kBK;
  }
  if (most < std::min(rows, kMinChunk)) return g;
  const int c0 = (rows + most - 1) / most;
  const uint64_t cap = debug_value(SYMPROP_DEBUG_GRAM_CHUNKS);  // 0: none
  double best = 1e300;
  for (int c = c0; c <= std::max(c0, std::min(c0 + 24, rows / kMinChunk)); ++c) {
    const int kc = ((rows + c - 1) / c + kBK - 1) / kBK * kBK;
    int group = c;
    while (group > 1 && bytes(kc, group) > limit) --group;
    // with the check among the sums' units (few = 0), or before them
    auto clocks = [&](int few) {
      double t = c * std::max(35000.0, 0.035 * cols * cols);
      auto launch = [&](double units, int kblocks) { t += std::ceil(units / n) * (kblocks * 1024.0 + 12000.0); };
      for (int x = 0; x < c; x += group) {
        const double part = (double)g.ntiles * std::min(group, c - x);
        launch(part * (few ? kP : planes), kc / kBK);
        if (few) launch(part, few), t += 60000.0;
      }
      return t;
    };
    for (int few : {0, planes > kP ? kc / kBK / 8 : 0}) {
      const double t = clocks(few);
      if (t < best) {
        best = t;
        g.nchunk = (rows + kc - 1) / kc;
        g.kc = kc;
        g.group = group;
        g.few = few;
      }
    }
  }
  g.chunk = (rows + g.nchunk - 1) / g.nchunk;  // chunks of like length: no short last one
  g.group = std::min(g.group, g.nchunk);
  if (cap) g.group = (int)std::min<uint64_t>(g.group, cap);
  g.res = res(g.kc, g.group);
  g.bytes = bytes(g.kc, g.group);
  return g;
}

}  // namespace

// Six launches, two waits and 256-wide tiles take 110 us and more, so that gemm's
// FP64 tiles win at odd widths of few rows (gram_f64, even widths, does not).  us, FP64
// kernel / this one with the check:
//   rows                     1,536      3,000      6,000      10,000     80,000
//   320 columns (even)     332 / 115  326 / 129  266 / 156  281 / 197  2,011 / 567
//   321 (odd)               66 / 119   96 / 132  175 / 146  257 / 181  1,934 / 557
//   513                    108 / 127  181 / 142  324 / 179  515 / 210  4,103 / 863
//   816                    337 / 157  333 / 182  277 / 235  438 / 304  3,209 / 1,363
//   2,002                  364 / 317  662 / 381  1,261 / 506  2,059 / 653  16,025 / 3,686
// The caller compares the two times (f64_gram_us in dense.cu).  This one is fitted to
// where they meet: over 190 sizes of 1,536 to 80,000 rows and 320 to 2,002 columns the
// faster kernel is taken at every one.  Below, only the FP64 kernels.
bool i8_gram_takes(int rows, int cols) { return cols >= 320 && rows >= 1536; }
double i8_gram_us(int rows, int cols) { return 70.0 + 0.002 * rows + 0.06 * cols + 1.5e-5 * rows * cols; }

// Entries that the caller of a componentwise Gram may have summed one by one: 64
// bytes of A a row each, against cols^2 / 2 FMAs a row for all of them by the FP64
// kernel (equal at about cols^2 / 900); a few odd columns always.
static unsigned max_pairs(int cols) {
  return (unsigned)std::max<long long>(4ll * cols, (long long)cols * cols / 1024);
}

bool gram_cols_i8(cudaStream_t st, const double *A, int rows, int cols, int lda, double *C, int ldc,
                  bool componentwise) {
  // the check of a componentwise Gram is one more plane of each chunk
  const int planes = kP + (componentwise ? 1 : 0);
  // operands of a launch: what the pool keeps (more, and not kept, from 16,641 columns
  // on, where the remainders alone pass that), less when the device has not that much left
  I8Plan g;
  std::optional<PoolBuf> ops;
  for (size_t limit = PoolBuf::kPoolMax; !ops; limit = g.bytes / 2) {
    g = plan_i8(rows, cols, planes, limit);
    if (!g.nchunk && limit == PoolBuf::kPoolMax) g = plan_i8(rows, cols, planes, 4 * limit);
    if (!g.nchunk) return false;
    try {
      ops.emplace(g.bytes, st);
    } catch (const Error &e) {
      if (e.code != SYMPROP_ERR_OOM) throw;
    }
  }
  signed char *const res = ops->as<signed char>();
  unsigned char *const rem = ops->as<unsigned char>() + g.res;
  const size_t ncs = (size_t)g.nchunk * cols;
  PoolBuf cmax(ncs * 8, st), sc(ncs * 4, st), flags(4 * sizeof(int), st);
  int *bad = (int *)flags.p, *err = bad + 1;
  SPB_CUDA(cudaMemsetAsync(cmax.p, 0, ncs * 8, st));
  SPB_CUDA(cudaMemsetAsync(flags.p, 0, 4 * sizeof(int), st));
  // a CTA walks its rows in 0.15 us each, so 8 CTAs an SM where there are rows for them
  // (512 rows a CTA: 80 us from 1,536 x 320 to 80,000 x 320)
  const int ctas = (cols + 127) / 128 * g.nchunk, parts = (8 * sms() + ctas - 1) / ctas,
            part = std::min(512, std::max(32, (g.chunk + parts - 1) / parts));
  col_max_kernel<<<dim3((cols + 127) / 128, g.nchunk, (g.chunk + part - 1) / part), 128, 0, st>>>(
      A, rows, cols, lda, g.chunk, part, (unsigned long long *)cmax.p);
  SPB_LAUNCH_CHECK();
  scale_kernel<<<(unsigned)((ncs + 255) / 256), 256, 0, st>>>((const unsigned long long *)cmax.p, (int)ncs,
                                                              (int *)sc.p, bad);
  SPB_LAUNCH_CHECK();
  int h[3] = {0, 0, 0};
  auto read_flags = [&] {  // false: A is left to the FP64 kernel
    SPB_CUDA(cudaMemcpyAsync(h, flags.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    SPB_CUDA(cudaStreamSynchronize(st));
    if (h[1]) fail(SYMPROP_ERR_TIMEOUT, "integer tensor-core Gram: a bounded wait expired");
    return !h[0] && (unsigned)h[2] <= max_pairs(cols);
  };
  if (!read_flags()) return false;
  PoolBuf list(componentwise ? max_pairs(cols) * sizeof(int2) : 0, st), nsq(componentwise ? ncs * 8 : 0, st);
  const Odd odd{list.as<int2>(), (unsigned *)(bad + 2), max_pairs(cols)};
  int *const suspect = bad + 3;
  if (componentwise) SPB_CUDA(cudaMemsetAsync(nsq.p, 0, ncs * 8, st));
  const size_t nblocks = g.few ? (size_t)g.group * (g.kc / kBK) : 0;
  PoolBuf blocks(nblocks * 8 + (size_t)g.group * g.few * sizeof(int), st);
  unsigned long long *const weight = g.few ? blocks.as<unsigned long long>() : nullptr;
  int *const picked = g.few ? reinterpret_cast<int *>(weight + nblocks) : nullptr;
  SPB_CUDA(cudaFuncSetAttribute(i8_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
  for (int c0 = 0; c0 < g.nchunk; c0 += g.group) {
    const int nc = std::min(g.group, g.nchunk - c0);
    if (g.few) SPB_CUDA(cudaMemsetAsync(weight, 0, nblocks * 8, st));
    auto residues = componentwise ? residue_kernel<true> : residue_kernel<false>;
    residues<<<dim3((cols + 31) / 32, g.kc / 128, nc), 128, 0, st>>>(A, rows, cols, lda, g.chunk, g.kc,
                                                                     (const int *)sc.p, c0, res,
                                                                     (unsigned long long *)nsq.p, weight, odd);
    SPB_LAUNCH_CHECK();
    CUtensorMap map;
    cuuint64_t dims[2] = {(cuuint64_t)g.kc, (cuuint64_t)nc * planes * cols};
    cuuint64_t strides[1] = {(cuuint64_t)g.kc};
    cuuint32_t box[2] = {kBK, kTile}, estr[2] = {1, 1};
    const CUresult r = get_encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, res, dims, strides, box, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) fail(SYMPROP_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    I8Args a{};
    a.cols = cols;
    a.ntile = g.ntile;
    a.ntiles = g.ntiles;
    a.C = rem;
    a.ld = g.ld;
    a.err = err;
    a.wait_ns = mainloop_wait_ns();
    a.expired_warp = expired_warp();
    a.planes = planes;
    a.nsq = (const unsigned long long *)nsq.p;
    a.chunk0 = c0;
    a.chunk = g.chunk;
    a.rows = rows;
    a.odd = odd;
    auto product = [&](int checks, bool sums, const int *picked = nullptr, int *suspect = nullptr) {
      a.checks = checks;
      a.some = picked != nullptr;
      a.suspect = suspect;
      a.picked = picked;
      a.kblocks = picked ? g.few : g.kc / kBK;
      i8_gram_kernel<<<(unsigned)(g.ntiles * (checks + (sums ? nc * kP : 0))), 256, kSmem, st>>>(map, a);
      SPB_LAUNCH_CHECK();
    };
    if (g.few) {
      pick_kernel<<<nc, 512, 0, st>>>(weight, g.kc / kBK, g.few, picked);
      SPB_LAUNCH_CHECK();
      product(nc, false, picked, suspect);
      product(nc, false, nullptr, suspect);
      product(0, true);
    } else {
      product(componentwise ? nc : 0, true);
    }
    const unsigned nt = (unsigned)((cols + 31) / 32);
    crt_kernel<<<dim3(nt, nt), 256, 0, st>>>(rem, g.ld, cols, nc, c0, (const int *)sc.p,
                                             c0 > 0 ? 1 : 0, C, ldc, odd);
    SPB_LAUNCH_CHECK();
  }
  if (!read_flags()) return false;
  if (h[2]) {
    pair_kernel<<<(unsigned)h[2], 256, 0, st>>>(odd.pairs, A, rows, lda, C, ldc);
    SPB_LAUNCH_CHECK();
  }
  return true;
}

}  // namespace gram
}  // namespace spb
