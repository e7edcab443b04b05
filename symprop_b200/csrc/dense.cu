// Dense steps of the Tucker loop on sm_100a (FP64 drop-in precision).
//
// Replaces the reference's CBLAS/LAPACKE wrappers
// (src/dense/matrixops.cpp): gemmtn (:45-56), symgemm (:102-124) and
// symsyrk (:126-146) become the tiled GEMM below; leftsvd (:18-43) and
// syevd (:77-100) become a block-Krylov top-r eigensolver on the packed Gram
// matrix with a one-CTA Jacobi for the projected problem; qr (:58-75)
// becomes CholQR2 with a Householder QR fallback.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "dense.cuh"
#include "gram_i8.cuh"

namespace spb {
namespace dense {

namespace {

inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// ------------------------------------------------------------------- GEMM

// 64 x NB tiles (NB = 64, or 32 for products of at most 32 columns), k blocks
// of 16 in two shared buffers: the next block's loads are in flight during the
// current one, one barrier per block.
constexpr int BM = 64, BK = 16;

template <typename T, int NB, bool TA, bool TB, bool KS>
__global__ void __launch_bounds__(256) gemm_tile_kernel(int M, int N, int K, const T *__restrict__ A,
                                                        int lda, const T *__restrict__ B, int ldb,
                                                        const T *__restrict__ ks, T *out, int ldo,
                                                        int kchunk, int sym_upper,
                                                        size_t split_stride) {
  const int tm = blockIdx.y, tn = blockIdx.x;
  if (sym_upper && tm * BM >= (tn + 1) * NB) return;  // below the diagonal
  constexpr int EA = BM * BK / 256, EB = NB * BK / 256, CN = NB / 16;
  const int bm = tm * BM, bn = tn * NB;
  const int k0 = blockIdx.z * kchunk;
  const int k1 = min(K, k0 + kchunk);
  __shared__ T As[2][BK][BM + 1];
  __shared__ T Bs[2][BK][NB + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  T ra[EA], rb[EB];
  auto fetch = [&](int kk) {
#pragma unroll
    for (int e = 0; e < EA; ++e) {
      const int idx = tid + e * 256, kq = TA ? idx / BM : idx % BK, im = TA ? idx % BM : idx / BK;
      const int gi = bm + im, gk = kk + kq;
      T v = T(0);
      if (gi < M && gk < k1) {
        v = TA ? A[(size_t)gk * lda + gi] : A[(size_t)gi * lda + gk];
        if (KS) v *= ks[gk];
      }
      ra[e] = v;
    }
#pragma unroll
    for (int e = 0; e < EB; ++e) {
      const int idx = tid + e * 256, kq = TB ? idx % BK : idx / NB, jn = TB ? idx / BK : idx % NB;
      const int gj = bn + jn, gk = kk + kq;
      rb[e] = gj < N && gk < k1 ? (TB ? B[(size_t)gj * ldb + gk] : B[(size_t)gk * ldb + gj]) : T(0);
    }
  };
  T acc[4][CN];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < CN; ++j) acc[i][j] = T(0);
  if (k0 < k1) fetch(k0);
  int buf = 0;
  for (int kk = k0; kk < k1; kk += BK, buf ^= 1) {
#pragma unroll
    for (int e = 0; e < EA; ++e) {
      const int idx = tid + e * 256;
      As[buf][TA ? idx / BM : idx % BK][TA ? idx % BM : idx / BK] = ra[e];
    }
#pragma unroll
    for (int e = 0; e < EB; ++e) {
      const int idx = tid + e * 256;
      Bs[buf][TB ? idx % BK : idx / NB][TB ? idx / BK : idx % NB] = rb[e];
    }
    __syncthreads();
    if (kk + BK < k1) fetch(kk + BK);
#pragma unroll
    for (int kq = 0; kq < BK; ++kq) {
      T a[4], b[CN];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[buf][kq][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < CN; ++j) b[j] = Bs[buf][kq][tx * CN + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) acc[i][j] += a[i] * b[j];
    }
  }
  T *o = out + blockIdx.z * split_stride;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gi = bm + ty * 4 + i;
    if (gi >= M) continue;
#pragma unroll
    for (int j = 0; j < CN; ++j) {
      int gj = bn + tx * CN + j;
      if (gj < N) o[(size_t)gi * ldo + gj] = acc[i][j];
    }
  }
}

// ------------------------------------------------ FP64 Gram C = A^T A
//
// The m x m Gram of the columns of a row-major n x m matrix (HOOI's dense
// step in FP64), upper tiles only: 128 x 128 tiles of C, 256 threads with
// 8 x 8 accumulators each (rows 32 q + 2 ty + {0, 1}, q < 4, the same for
// the columns with tx: a warp's 16-byte loads of one k row are then
// contiguous and free of bank conflicts), k-blocks of 16 rows of A staged in shared
// memory by cp.async in a 3-stage ring.  The K axis is cut into splits
// whose partial tiles the finalize kernel adds (and mirrors).
constexpr int GB = 128, GK = 16, GST = 3;

struct GramSmem {
  double a[GST][GK][GB];
  double b[GST][GK][GB];
};

__device__ __forceinline__ void cp_async16_zfill(void *dst, const void *src, bool full) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int sz = full ? 16 : 0;  // 0: fill the 16 bytes with zeros, read nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
}

__global__ void __launch_bounds__(256, 1) gram_tn_f64_kernel(int M, int K, const double *__restrict__ A, int lda,
                                                             int ntile, int kchunk, double *out,
                                                             size_t split_stride) {
  extern __shared__ __align__(16) unsigned char gram_raw[];
  GramSmem &sm = *reinterpret_cast<GramSmem *>(gram_raw);
  // upper tile (ti, tj), ti <= tj, of linear index blockIdx.x (row by row)
  int ti = 0, rem = (int)blockIdx.x;
  while (rem >= ntile - ti) {
    rem -= ntile - ti;
    ++ti;
  }
  const int tj = ti + rem;
  const bool diag = ti == tj;
  const int i0 = ti * GB, j0 = tj * GB;
  const int k0 = (int)blockIdx.y * kchunk, k1 = min(K, k0 + kchunk);
  const int nkb = (k1 - k0 + GK - 1) / GK;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;

  auto load = [&](int kb, int stage) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = tid + 256 * q, kr = c >> 6, col = (c & 63) * 2;
      const int gk = k0 + kb * GK + kr;
      const bool oka = gk < k1 && i0 + col < M;
      cp_async16_zfill(&sm.a[stage][kr][col], oka ? A + (size_t)gk * lda + i0 + col : A, oka);
      if (!diag) {
        const bool okb = gk < k1 && j0 + col < M;
        cp_async16_zfill(&sm.b[stage][kr][col], okb ? A + (size_t)gk * lda + j0 + col : A, okb);
      }
    }
  };
#pragma unroll
  for (int s = 0; s < GST - 1; ++s) {
    if (s < nkb) load(s, s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  double acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
  for (int kb = 0; kb < nkb; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GST - 2) : "memory");
    __syncthreads();
    if (kb + GST - 1 < nkb) load(kb + GST - 1, (kb + GST - 1) % GST);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int stg = kb % GST;
    const double(*As)[GB] = sm.a[stg];
    const double(*Bs)[GB] = diag ? sm.a[stg] : sm.b[stg];
#pragma unroll 4
    for (int kk = 0; kk < GK; ++kk) {
      double a[8], b[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double2 av = *reinterpret_cast<const double2 *>(&As[kk][32 * q + 2 * ty]);
        const double2 bv = *reinterpret_cast<const double2 *>(&Bs[kk][32 * q + 2 * tx]);
        a[2 * q] = av.x, a[2 * q + 1] = av.y;
        b[2 * q] = bv.x, b[2 * q + 1] = bv.y;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  double *o = out + blockIdx.y * split_stride;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gi = i0 + 32 * (i >> 1) + 2 * ty + (i & 1);
    if (gi >= M) continue;
#pragma unroll
    for (int jh = 0; jh < 4; ++jh) {
      const int gj = j0 + 32 * jh + 2 * tx;
      if (gj < M) *reinterpret_cast<double2 *>(&o[(size_t)gi * M + gj]) = make_double2(acc[i][2 * jh], acc[i][2 * jh + 1]);
    }
  }
}

// ------------------------------------ FP64 panel W = A diag(ks) B, N <= 16
//
// HOOI's U = Y D^1/2 V and HOQRI's Y D C^T in FP64: a tall row-major A
// (M x K) times a K x N matrix with N <= 16.  One CTA of 256 threads per 64
// rows of A, K in blocks of 32 (the A block read once, coalesced along k;
// the scaled B block broadcast from shared memory); each thread keeps 4
// outputs (row tid / 4, columns 4 (tid % 4) .. + 3).  HBM-bound on A.
constexpr int PR = 64, PK = 32;

__global__ void __launch_bounds__(256) panel_f64_kernel(int M, int N, int K, const double *__restrict__ A, int lda,
                                                        const double *__restrict__ B, int ldb, bool transB,
                                                        const double *__restrict__ ks, double *__restrict__ W,
                                                        int ldw) {
  __shared__ double As[PR][PK + 1];
  __shared__ __align__(16) double Bs[PK][16];
  const int tid = threadIdx.x, row = tid >> 2, c0 = (tid & 3) * 4;
  const int i0 = blockIdx.x * PR;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int k0 = 0; k0 < K; k0 += PK) {
    double av[PR * PK / 256];
#pragma unroll
    for (int t = 0; t < PR * PK / 256; ++t) {
      const int e = tid + 256 * t, ii = e / PK, kk = e % PK, gi = i0 + ii, gk = k0 + kk;
      av[t] = gi < M && gk < K ? A[(size_t)gi * lda + gk] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < PR * PK / 256; ++t) {
      const int e = tid + 256 * t;
      As[e / PK][e % PK] = av[t];
    }
    for (int e = tid; e < PK * 16; e += 256) {
      const int kk = e >> 4, q = e & 15, gk = k0 + kk;
      double b = 0.0;
      if (gk < K && q < N) {
        b = transB ? B[(size_t)q * ldb + gk] : B[(size_t)gk * ldb + q];
        if (ks) b *= ks[gk];
      }
      Bs[kk][q] = b;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < PK; ++kk) {
      const double a = As[row][kk];
      const double2 b0 = *reinterpret_cast<const double2 *>(&Bs[kk][c0]);
      const double2 b1 = *reinterpret_cast<const double2 *>(&Bs[kk][c0 + 2]);
      acc[0] = fma(a, b0.x, acc[0]);
      acc[1] = fma(a, b0.y, acc[1]);
      acc[2] = fma(a, b1.x, acc[2]);
      acc[3] = fma(a, b1.y, acc[3]);
    }
    __syncthreads();
  }
  const int gi = i0 + row;
  if (gi < M)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c0 + j < N) W[(size_t)gi * ldw + c0 + j] = acc[j];
}

// C = alpha * sum_z P[z] + beta * C, mirroring the lower triangle for sym_upper
template <typename T>
__global__ void gemm_finalize_kernel(int M, int N, const T *P, int splits, size_t stride, T alpha,
                                     T beta, T *C, int ldc, int sym_upper) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)M * N) return;
  int i = (int)(idx / N), j = (int)(idx % N);
  int si = i, sj = j;
  if (sym_upper && (i / BM) > (j / BM)) { si = j; sj = i; }
  T s = T(0);
  for (int z = 0; z < splits; ++z) s += P[z * stride + (size_t)si * N + sj];
  T prev = beta != T(0) ? C[(size_t)i * ldc + j] : T(0);
  C[(size_t)i * ldc + j] = alpha * s + beta * prev;
}

// --------------------------------------------------------- reductions

constexpr int kRedBlocks = 296;

template <typename T>
__global__ void wsq_partial_kernel(const T *X, const T *Y, const double *w, int rows, int cols,
                                   double *part) {
  double a = 0.0, b = 0.0;
  size_t total = (size_t)rows * cols;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    int q = (int)(idx % cols);
    double x = (double)X[idx];
    double d = x - (Y ? (double)Y[idx] : 0.0);
    double ww = w ? w[q] : 1.0;
    a += ww * d * d;
    b += ww * x * x;
  }
  __shared__ double sa[256], sb[256];
  sa[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sa[threadIdx.x] += sa[threadIdx.x + s];
      sb[threadIdx.x] += sb[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sa[0];
    part[2 * blockIdx.x + 1] = sb[0];
  }
}

__global__ void sum_pairs_kernel(const double *part, int n, double *out) {
  __shared__ double sa[256], sb[256];
  double a = 0, b = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    a += part[2 * i];
    b += part[2 * i + 1];
  }
  sa[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sa[threadIdx.x] += sa[threadIdx.x + s];
      sb[threadIdx.x] += sb[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = sa[0];
    out[1] = sb[0];
  }
}

// ------------------------------------------------------------ Cholesky

// G (c x c) -> Rinv with A Rinv orthonormal for G = A^T A.  The columns are
// first scaled to unit norm (G' = D G D, D = diag(G)^-1/2), so the pivot test
// measures linear dependence, not column scaling; Rinv = D R'^-1 with
// G' = R'^T R'.  status[0] = 1 when a pivot is not safely positive.
__global__ void chol_inv_kernel(const double *G, int c, double *Rinv, int *status) {
  extern __shared__ double sm[];
  double *R = sm;          // c x c
  double *Ri = sm + c * c; // c x c
  __shared__ double dsc[64];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < c; i += nt) {
    double g = G[i * c + i];
    dsc[i] = g > 0 ? 1.0 / sqrt(g) : 1.0;
  }
  __syncthreads();
  for (int i = tid; i < c * c; i += nt) {
    R[i] = G[i] * dsc[i / c] * dsc[i % c];
    Ri[i] = 0.0;
  }
  __syncthreads();
  __shared__ double maxd;
  __shared__ int bad;
  if (tid == 0) {
    maxd = 0;
    bad = 0;
    for (int i = 0; i < c; ++i) maxd = fmax(maxd, fabs(R[i * c + i]));
  }
  __syncthreads();
  // right-looking Cholesky on the upper triangle: R[k][k..] row k of R
  for (int k = 0; k < c; ++k) {
    if (tid == 0) {
      double d = R[k * c + k];
      if (!(d > 1e-13 * maxd) || !(maxd > 0)) {
        bad = 1;
        d = fmax(fabs(d), 1e-300);
      }
      R[k * c + k] = sqrt(d);
    }
    __syncthreads();
    double rkk = R[k * c + k];
    for (int j = k + 1 + tid; j < c; j += nt) R[k * c + j] /= rkk;
    __syncthreads();
    for (int idx = tid; idx < c * c; idx += nt) {
      int i = idx / c, j = idx % c;
      if (i > k && j >= i) R[i * c + j] -= R[k * c + i] * R[k * c + j];
    }
    __syncthreads();
  }
  // inverse of upper-triangular R: column by column back substitution
  for (int j = tid; j < c; j += nt) {
    for (int i = j; i >= 0; --i) {
      double s = (i == j) ? 1.0 : 0.0;
      for (int k = i + 1; k <= j; ++k) s -= R[i * c + k] * Ri[k * c + j];
      Ri[i * c + j] = s / R[i * c + i];
    }
  }
  __syncthreads();
  for (int i = tid; i < c * c; i += nt) Rinv[i] = Ri[i] * dsc[i / c];
  if (tid == 0) status[0] = bad;
}

// The same for c <= C (16 or 32) by one warp: lane j holds column j, rows
// unrolled, so a step is a shared (broadcast) load and an FMA per row instead of
// three barriers (c = 32: 37 -> 23 us, c = 16: 16.5 -> 6.8 us).  Lanes and rows
// from c on hold the identity.
template <int C>
__global__ void __launch_bounds__(32) chol_inv_warp_kernel(const double *G, int c, double *Rinv, int *status) {
  const int j = threadIdx.x;
  const bool in = j < c;
  const double gjj = in ? G[j * c + j] : 1.0;
  const double d = gjj > 0.0 ? 1.0 / sqrt(gjj) : 1.0;
  __shared__ __align__(16) double R[C][C];
  double r[C], x[C], ri[C];  // column j of R and of its inverse, 1 / diagonal of R
  double maxd = in ? fabs(gjj * d * d) : 0.0;
#pragma unroll
  for (int i = 0; i < C; ++i) {
    const double di = __shfl_sync(0xffffffffu, d, i);
    r[i] = in && i < c ? G[i * c + j] * di * d : i == j ? 1.0 : 0.0;
  }
  for (int o = 16; o > 0; o >>= 1) maxd = fmax(maxd, __shfl_xor_sync(0xffffffffu, maxd, o));
  bool bad = false;
#pragma unroll
  for (int k = 0; k < C; ++k) {
    double p = __shfl_sync(0xffffffffu, r[k], k);
    if (k < c && (!(p > 1e-13 * maxd) || !(maxd > 0.0))) {
      bad = true;
      p = fmax(fabs(p), 1e-300);
    }
    const double root = sqrt(p);
    ri[k] = 1.0 / root;
    r[k] = j == k ? root : r[k] * ri[k];
    if (j < C) R[k][j] = r[k];
    __syncwarp();
#pragma unroll
    for (int i = k + 1; i < C; ++i) r[i] = fma(-R[k][i], r[k], r[i]);
  }
  // R x = e_j by back substitution (x_i = 0 for i > j)
#pragma unroll
  for (int i = C - 1; i >= 0; --i) {
    double s = i == j ? 1.0 : 0.0;
#pragma unroll
    for (int k = i + 1; k < C; ++k) s = fma(-R[i][k], x[k], s);
    x[i] = i <= j ? s * ri[i] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < C; ++i) {
    const double di = __shfl_sync(0xffffffffu, d, i);
    if (in && i < c) Rinv[i * c + j] = x[i] * di;
  }
  if (j == 0) status[0] = bad;
}

// ---------------------------------------------------- Householder (1 CTA)

// deterministic block reduction (warp shuffles, fixed tree); red >= 33 doubles
__device__ double block_sum(double v, double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double w = lane < nw ? red[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
    if (lane == 0) red[32] = w;
  }
  __syncthreads();
  double r = red[32];
  __syncthreads();
  return r;
}

// A (rows x c) -> explicit Q as dgeqrf + dorgqr; v vectors kept in A,
// Q built in Qout.  One CTA of 1024 threads; used for rank-deficient inputs.
__global__ void __launch_bounds__(1024) householder_kernel(double *A, int rows, int c, double *tau,
                                                           double *Q) {
  __shared__ double red[1024];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int j = 0; j < c && j < rows; ++j) {
    double s = 0;
    for (int i = j + 1 + tid; i < rows; i += nt) s += A[(size_t)i * c + j] * A[(size_t)i * c + j];
    double sigma = block_sum(s, red);
    double alpha = A[(size_t)j * c + j];
    double t = 0, beta = alpha;
    if (sigma > 0) {
      beta = -copysign(sqrt(alpha * alpha + sigma), alpha);
      t = (beta - alpha) / beta;
      double scal = 1.0 / (alpha - beta);
      for (int i = j + 1 + tid; i < rows; i += nt) A[(size_t)i * c + j] *= scal;
    }
    __syncthreads();
    if (tid == 0) {
      tau[j] = t;
      A[(size_t)j * c + j] = beta;
    }
    __syncthreads();
    // apply H = I - t v v^T to columns j+1..c-1 (v[j] = 1)
    for (int k = j + 1; k < c; ++k) {
      double w = 0;
      for (int i = j + tid; i < rows; i += nt) {
        double v = (i == j) ? 1.0 : A[(size_t)i * c + j];
        w += v * A[(size_t)i * c + k];
      }
      w = block_sum(w, red);
      for (int i = j + tid; i < rows; i += nt) {
        double v = (i == j) ? 1.0 : A[(size_t)i * c + j];
        A[(size_t)i * c + k] -= t * v * w;
      }
      __syncthreads();
    }
  }
  // Q = H_0 ... H_{c-1} [I; 0]
  for (size_t idx = tid; idx < (size_t)rows * c; idx += nt) {
    size_t i = idx / c, k = idx % c;
    Q[idx] = (i == k) ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int j = min(c, rows) - 1; j >= 0; --j) {
    double t = tau[j];
    for (int k = j; k < c; ++k) {
      double w = 0;
      for (int i = j + tid; i < rows; i += nt) {
        double v = (i == j) ? 1.0 : A[(size_t)i * c + j];
        w += v * Q[(size_t)i * c + k];
      }
      w = block_sum(w, red);
      for (int i = j + tid; i < rows; i += nt) {
        double v = (i == j) ? 1.0 : A[(size_t)i * c + j];
        Q[(size_t)i * c + k] -= t * v * w;
      }
      __syncthreads();
    }
  }
}

// --------------------------------------------------------------- Jacobi

// Cyclic Jacobi with the round-robin pairing (np - 1 steps of np / 2 disjoint
// pairs a sweep), in two kernels:
//   jacobi_kernel  one CTA: the upper triangle of A in shared memory.  Per step
//                  np / 2 threads form the rotations, then a thread per pair of
//                  rotations (k <= l) updates the 2 x 2 block of A that they
//                  share, rows and columns at once: two barriers a step.  The
//                  rotations go to memory.
//   jacobi_vectors_kernel  V = product of the rotations: its rows are
//                  independent, one warp each.
// Bound by latency: a step is a chain of a few hundred cycles (rotation,
// barrier, block, barrier) whatever n is.  n = 96: 2.75 ms with rows,
// columns and V updated in turn by one CTA (four barriers a step, a serial
// sort), 0.92 + 0.19 ms now; n = 64: 1.04 -> 0.39 + 0.09 ms.
constexpr int kJacobiSweeps = 60;

// the pair of place k at a step: indices p < q
__device__ __forceinline__ void jacobi_pair(int k, int step, int np, int &p, int &q) {
  int a = k + step;  // 1 + (k - 1 + step) mod (np - 1), k >= 1
  a = k == 0 ? 0 : a >= np ? a - (np - 1) : a;
  int b = np - 1 - k + step;
  b = b >= np ? b - (np - 1) : b;
  p = min(a, b);
  q = max(a, b);
}

// w_out: eigenvalues, descending; place[j]: place of index j among them;
// rot: (c, s) of every pair of every step; *sweeps: how many were done
__global__ void __launch_bounds__(1024) jacobi_kernel(const double *S, int n, double *w_out, double2 *rot, int *place,
                                                      int *sweeps) {
  extern __shared__ double A[];  // np x ld, upper triangle
  const int np = (n + 1) & ~1, half = np / 2;
  const int ld = np + 1;  // odd row stride: column reads fall on different banks
  __shared__ double2 cs[kJacobiMax / 2];
  __shared__ int2 pr[kJacobiMax / 2];
  __shared__ double red[33];
  __shared__ int rotated;
  const int tid = threadIdx.x, nt = blockDim.x;
  // scaled by a power of two to entries of at most 1
  double mx = 0.0;
  for (int idx = tid; idx < n * n; idx += nt) mx = fmax(mx, fabs(S[idx]));
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) red[tid >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < nt / 32; ++w) mx = fmax(mx, red[w]);
  __syncthreads();
  int e = 0;
  if (mx > 0.0 && isfinite(mx)) frexp(mx, &e);
  double fro = 0.0;
  for (int idx = tid; idx < np * np; idx += nt) {
    const int i = idx / np, j = idx % np;
    const double x = i < n && j < n ? scalbn(S[i * n + j], -e) : 0.0;
    fro += x * x;
    if (i <= j) A[i * ld + j] = x;
  }
  fro = block_sum(fro, red);
  const double tiny = 1e-18 * sqrt(fro);
  // this thread's blocks: pairs (k, l) of rotations, k <= l
  constexpr int kBlk = 2;  // 48 * 49 / 2 over at least 588 threads
  const int nblk = half * (half + 1) / 2;
  int bk[kBlk], bl[kBlk];
#pragma unroll
  for (int t = 0; t < kBlk; ++t) {
    int k = 0, r = tid + t * nt;
    bk[t] = -1;
    bl[t] = 0;
    if (r < nblk) {
      while (r >= half - k) {
        r -= half - k;
        ++k;
      }
      bk[t] = k;
      bl[t] = k + r;
    }
  }
  int sweep = 0;
  for (; sweep < kJacobiSweeps && np > 1; ++sweep) {
    double off = 0.0;
    for (int idx = tid; idx < np * np; idx += nt) {
      const int i = idx / np, j = idx % np;
      if (i < j) off += A[i * ld + j] * A[i * ld + j];
    }
    off = 2.0 * block_sum(off, red);
    if (!(off > 1e-30 * fro)) break;
    if (tid == 0) rotated = 0;
    __syncthreads();
    for (int step = 0; step < np - 1; ++step) {
      if (tid < half) {
        int p, q;
        jacobi_pair(tid, step, np, p, q);
        const double apq = A[p * ld + q], app = A[p * ld + p], aqq = A[q * ld + q];
        double c = 1.0, sn = 0.0;
        // an element below the rounding level of its diagonal pair (or of
        // the whole matrix) is left alone; a sweep that rotates nothing ends
        // the iteration (rounding noise keeps off() from reaching zero)
        if (!(apq * apq <= 1e-34 * fabs(app * aqq) || fabs(apq) <= tiny)) {
          rotated = 1;
          // the tangent needs few digits (what it leaves of apq, 1e-7 of it, is
          // the next sweep's); the rotation must be orthogonal to the last one
          const float tau = (float)(aqq - app) / (float)(2.0 * apq);
          const double t = (double)((tau >= 0.f ? 1.f : -1.f) / (fabsf(tau) + sqrtf(1.f + tau * tau)));
          c = rsqrt(fma(t, t, 1.0));
          sn = t * c;
        }
        cs[tid] = make_double2(c, sn);
        pr[tid] = make_int2(p, q);
        rot[((size_t)sweep * (np - 1) + step) * half + tid] = make_double2(c, sn);
      }
      __syncthreads();
#pragma unroll
      for (int t = 0; t < kBlk; ++t) {
        if (bk[t] < 0) continue;
        const double2 u = cs[bk[t]], v = cs[bl[t]];
        if (u.y == 0.0 && v.y == 0.0) continue;
        const int2 r = pr[bk[t]], c = pr[bl[t]];
        double *x00 = A + min(r.x, c.x) * ld + max(r.x, c.x), *x01 = A + min(r.x, c.y) * ld + max(r.x, c.y),
               *x10 = A + min(r.y, c.x) * ld + max(r.y, c.x), *x11 = A + min(r.y, c.y) * ld + max(r.y, c.y);
        const double a00 = *x00, a01 = *x01, a10 = *x10, a11 = *x11;
        const double b00 = u.x * a00 - u.y * a10, b01 = u.x * a01 - u.y * a11;  // rows
        const double b10 = u.y * a00 + u.x * a10, b11 = u.y * a01 + u.x * a11;
        *x00 = v.x * b00 - v.y * b01;  // columns
        *x01 = v.y * b00 + v.x * b01;
        if (bk[t] != bl[t]) *x10 = v.x * b10 - v.y * b11;  // (k, k): the mirror image of x01
        *x11 = v.y * b10 + v.x * b11;
      }
      __syncthreads();
    }
    if (rotated == 0) {
      ++sweep;
      break;
    }
  }
  // eigenvalues descending (only the first n indices are real)
  if (tid == 0) *sweeps = sweep;
  auto key = [&](int j) {  // orders as the value, NaNs included
    const long long b = __double_as_longlong(A[j * ld + j]);
    return b < 0 ? ~(unsigned long long)b : (unsigned long long)b | 0x8000000000000000ull;
  };
  for (int j = tid; j < n; j += nt) {
    const unsigned long long x = key(j);
    int r = 0;
    for (int i = 0; i < n; ++i) {
      const unsigned long long y = key(i);
      r += y > x || (y == x && i < j);
    }
    place[j] = r;
    w_out[r] = scalbn(A[j * ld + j], e);
  }
}

// Row blockIdx.x of V = I J_1 J_2 ..., columns at their places
__global__ void __launch_bounds__(32) jacobi_vectors_kernel(const double2 *rot, const int *place, const int *sweeps,
                                                            int n, double *V_out) {
  __shared__ double v[kJacobiMax];
  const int np = (n + 1) & ~1, half = np / 2, lane = threadIdx.x, row = blockIdx.x;
  for (int j = lane; j < np; j += 32) v[j] = j == row ? 1.0 : 0.0;
  __syncwarp();
  const int steps = *sweeps * (np - 1);
  constexpr int kPer = (kJacobiMax / 2 + 31) / 32, kAhead = 8;  // steps in flight
  auto fetch = [&](int t, double2 (&r)[kPer]) {
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      r[i] = t < steps && lane + 32 * i < half ? rot[(size_t)t * half + lane + 32 * i] : make_double2(1.0, 0.0);
  };
  double2 nx[kAhead][kPer];
#pragma unroll
  for (int a = 0; a < kAhead; ++a) fetch(a, nx[a]);
  for (int t0 = 0, step = 0; t0 < steps; t0 += kAhead) {
#pragma unroll
    for (int a = 0; a < kAhead; ++a) {  // the steps past the last are identities
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const double2 r = nx[a][i];
        if (lane + 32 * i < half && r.y != 0.0) {
          int p, q;
          jacobi_pair(lane + 32 * i, step, np, p, q);
          const double x = v[p], y = v[q];
          v[p] = r.x * x - r.y * y;
          v[q] = r.y * x + r.x * y;
        }
      }
      fetch(t0 + kAhead + a, nx[a]);
      __syncwarp();
      step = step + 1 == np - 1 ? 0 : step + 1;
    }
  }
  for (int j = lane; j < n; j += 32) V_out[(size_t)row * n + place[j]] = v[j];
}

// ------------------------------------------------------------- misc

__global__ void scale_sym_kernel(double *G, int m, const double *sd) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)m * m) return;
  int i = (int)(idx / m), j = (int)(idx % m);
  G[idx] *= sd[i] * sd[j];
}

__global__ void clip_rows_kernel(double *U, int n, int r, double delta) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0;
  for (int j = 0; j < r; ++j) s += U[(size_t)i * r + j] * U[(size_t)i * r + j];
  s = sqrt(s);
  if (delta < s) {  // src/sparse/spsymtensor.cpp:172-183
    double mul = delta / s;
    for (int j = 0; j < r; ++j) U[(size_t)i * r + j] *= mul;
  }
}

template <typename Ts, typename Td>
__global__ void convert_kernel(const Ts *a, Td *b, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (Td)a[i];
}

__global__ void random_fill_kernel(double *A, size_t n, uint64_t seed) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t z = seed + 0x9E3779B97F4A7C15ull * (i + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  A[i] = ((double)(z >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
}

__global__ void eye_kernel(double *I, int s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < s) I[(size_t)i * s + i] = 1.0;
}

__global__ void copy_cols_kernel(const double *src, int lds, int rows, int cols, double *dst,
                                 int ldd) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)rows * cols) return;
  int i = (int)(idx / cols), j = (int)(idx % cols);
  dst[(size_t)i * ldd + j] = src[(size_t)i * lds + j];
}

// residual norms ||S x_i - lam_i x_i|| for i < r
__global__ void residual_kernel(const double *SX, const double *X, int s, int ld, int r,
                                const double *lam, double *res) {
  __shared__ double red[256];
  int i = blockIdx.x;
  double acc = 0;
  for (int row = threadIdx.x; row < s; row += blockDim.x) {
    double d = SX[(size_t)row * ld + i] - lam[i] * X[(size_t)row * ld + i];
    acc += d * d;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) res[i] = sqrt(red[0]);
}

using Scratch = PoolBuf;

// Partial core products P[chunk][q][j] = sum_{i in chunk} U[i][q0 + q] Y[i][j]
// over FP32 Y (n x m, read once, coalesced along j) and FP64 U (n x r): one
// thread per column j, kCoreRB FP64 accumulators, the U rows of the chunk
// staged in shared memory 64 at a time (every thread reads the same entry).
constexpr int kCoreRB = 16, kCoreRows = 64;
template <typename TY>
__global__ void __launch_bounds__(128) core_partial_kernel(const double *__restrict__ U,
                                                           const TY *__restrict__ Y, int n, int m,
                                                           int r, int q0, int rows_per_chunk,
                                                           double *__restrict__ P) {
  __shared__ double Us[kCoreRows][kCoreRB];
  const int col = blockIdx.x * 128 + threadIdx.x;
  const int i0 = blockIdx.y * rows_per_chunk, i1 = min(n, i0 + rows_per_chunk);
  double acc[kCoreRB];
#pragma unroll
  for (int q = 0; q < kCoreRB; ++q) acc[q] = 0.0;
  for (int ib = i0; ib < i1; ib += kCoreRows) {
    for (int t = threadIdx.x; t < kCoreRows * kCoreRB; t += 128) {
      const int ii = t / kCoreRB, q = t % kCoreRB;
      Us[ii][q] = (ib + ii < i1 && q0 + q < r) ? U[(size_t)(ib + ii) * r + q0 + q] : 0.0;
    }
    __syncthreads();
    const int cnt = min(kCoreRows, i1 - ib);
    if (col < m) {
      for (int ii = 0; ii < cnt; ++ii) {
        const double y = (double)Y[(size_t)(ib + ii) * m + col];
#pragma unroll
        for (int q = 0; q < kCoreRB; ++q) acc[q] = fma(Us[ii][q], y, acc[q]);
      }
    }
    __syncthreads();
  }
  if (col < m) {
#pragma unroll
    for (int q = 0; q < kCoreRB; ++q) P[((size_t)blockIdx.y * kCoreRB + q) * m + col] = acc[q];
  }
}

// core[q0 + q][j] = sum over chunks (in chunk order) of P[chunk][q][j]
__global__ void core_reduce_kernel(const double *__restrict__ P, int chunks, int m, int r, int q0,
                                   double *__restrict__ core) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)kCoreRB * m) return;
  const int q = (int)(idx / m), j = (int)(idx % m);
  if (q0 + q >= r) return;
  double s = 0.0;
  for (int c = 0; c < chunks; ++c) s += P[((size_t)c * kCoreRB + q) * m + j];
  core[(size_t)(q0 + q) * m + j] = s;
}

}  // namespace

// ------------------------------------------------------------ public API

// Tiles and K splits of gram_f64: the fewest splits (each at least 1024 rows)
// that fill 90% of the waves of one CTA per SM.
struct GramSplits {
  int nt, splits, kchunk;
  long long tiles, waves;
};

static GramSplits gram_splits(int M, int K) {
  static int nsm = 0;
  if (!nsm) {
    int dev = 0;
    SPB_CUDA(cudaGetDevice(&dev));
    SPB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  }
  GramSplits g;
  g.nt = (M + GB - 1) / GB;
  g.tiles = (long long)g.nt * (g.nt + 1) / 2;
  g.splits = 1;
  for (int s = 1; s <= 8; ++s) {
    if (s > 1 && K / s < 1024) break;
    const long long ctas = g.tiles * s, waves = (ctas + nsm - 1) / nsm;
    g.splits = s;
    if ((double)ctas >= 0.9 * (double)(waves * nsm)) break;
  }
  g.kchunk = (int)(cdiv(cdiv(K, g.splits), GK) * GK);
  g.splits = std::max(1, (int)cdiv(K, g.kchunk));
  g.waves = (g.tiles * g.splits + nsm - 1) / nsm;
  return g;
}

static bool gram_f64_takes(int M, const double *A, int lda) {
  return M >= GB && M % 2 == 0 && lda % 2 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
}

// C = A^T A (upper tiles computed, the rest mirrored) for a row-major
// K x M matrix A; M even, lda even, A 16-byte aligned.
static void gram_f64(cudaStream_t st, int M, int K, const double *A, int lda, double *C, int ldc) {
  const GramSplits g = gram_splits(M, K);
  const int nt = g.nt, splits = g.splits, kchunk = g.kchunk;
  const long long tiles = g.tiles;
  Scratch ws(sizeof(double) * (size_t)splits * M * M, st);
  const size_t smem = sizeof(GramSmem);
  SPB_CUDA(cudaFuncSetAttribute(gram_tn_f64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  gram_tn_f64_kernel<<<dim3((unsigned)tiles, (unsigned)splits), 256, smem, st>>>(M, K, A, lda, nt, kchunk,
                                                                                 ws.as<double>(), (size_t)M * M);
  SPB_LAUNCH_CHECK();
  gemm_finalize_kernel<double><<<cdiv((long long)M * M, 256), 256, 0, st>>>(M, M, ws.as<double>(), splits,
                                                                           (size_t)M * M, 1.0, 0.0, C, ldc, 1);
  SPB_LAUNCH_CHECK();
}

template <typename T>
void gemm(cudaStream_t st, int M, int N, int K, T alpha, const T *A, int lda, bool transA,
          const T *B, int ldb, bool transB, T beta, T *C, int ldc, const T *kscale,
          bool sym_upper) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0) {
    if (beta == T(0)) {
      for (int i = 0; i < M; ++i) SPB_CUDA(cudaMemsetAsync(C + (size_t)i * ldc, 0, N * sizeof(T), st));
      return;
    }
  }
  if constexpr (std::is_same<T, double>::value) {
    if (!transA && !sym_upper && N <= 16 && M >= 4 * PR && alpha == 1.0 && beta == 0.0) {
      panel_f64_kernel<<<cdiv(M, PR), 256, 0, st>>>(M, N, K, A, lda, B, ldb, transB, kscale, C, ldc);
      SPB_LAUNCH_CHECK();
      return;
    }
    if (transA && !transB && sym_upper && A == B && lda == ldb && M == N && !kscale && gram_f64_takes(M, A, lda) &&
        alpha == 1.0 && beta == 0.0) {
      gram_f64(st, M, K, A, lda, C, ldc);
      return;
    }
  }
  const int nb = N <= 32 && !sym_upper ? 32 : 64;
  const int tm = cdiv(M, BM), tn = cdiv(N, nb);
  long long tiles = sym_upper ? (long long)tm * (tm + 1) / 2 : (long long)tm * tn;
  // K splits up to two CTAs per SM, each of at least 4 k blocks (8 where the
  // partial sums to be added would be many): a block costs about 0.6 us whatever
  // the tile, and the eigensolver's products of a few tiles and K = 250 or 3,876
  // took 45 us with splits of at least 256
  int splits = (int)std::max<long long>(1, std::min<long long>((296 + tiles - 1) / tiles, cdiv(K, K > 1024 ? 128 : 64)));
  int kchunk = (int)(cdiv(cdiv(K, splits), BK) * BK);
  splits = std::max(1, (int)cdiv(K, kchunk));
  const bool direct = splits == 1 && alpha == T(1) && beta == T(0) && !sym_upper;
  Scratch ws(direct ? 0 : (size_t)splits * M * N * sizeof(T), st);
  T *out = direct ? C : ws.as<T>();
  const int ldo = direct ? ldc : N;
  const size_t stride = (size_t)M * N;
  dim3 grid(tn, tm, splits);
#define SPB_GEMM_LAUNCH(TA, TB, KS)                                                                          \
  do {                                                                                                       \
    if (nb == 32)                                                                                            \
      gemm_tile_kernel<T, 32, TA, TB, KS><<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, kscale, out, ldo,   \
                                                                kchunk, 0, stride);                          \
    else                                                                                                     \
      gemm_tile_kernel<T, 64, TA, TB, KS><<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, kscale, out, ldo,   \
                                                                kchunk, sym_upper ? 1 : 0, stride);          \
  } while (0)
  const bool ks = kscale != nullptr;
  if (transA && transB) { if (ks) SPB_GEMM_LAUNCH(true, true, true); else SPB_GEMM_LAUNCH(true, true, false); }
  else if (transA) { if (ks) SPB_GEMM_LAUNCH(true, false, true); else SPB_GEMM_LAUNCH(true, false, false); }
  else if (transB) { if (ks) SPB_GEMM_LAUNCH(false, true, true); else SPB_GEMM_LAUNCH(false, true, false); }
  else { if (ks) SPB_GEMM_LAUNCH(false, false, true); else SPB_GEMM_LAUNCH(false, false, false); }
#undef SPB_GEMM_LAUNCH
  SPB_LAUNCH_CHECK();
  if (!direct) {
    gemm_finalize_kernel<T><<<cdiv((long long)M * N, 256), 256, 0, st>>>(
        M, N, out, splits, stride, alpha, beta, C, ldc, sym_upper ? 1 : 0);
    SPB_LAUNCH_CHECK();
  }
}

template void gemm<double>(cudaStream_t, int, int, int, double, const double *, int, bool,
                           const double *, int, bool, double, double *, int, const double *, bool);
template void gemm<float>(cudaStream_t, int, int, int, float, const float *, int, bool,
                          const float *, int, bool, float, float *, int, const float *, bool);

template <typename TY>
static void core_from(cudaStream_t st, const double *U, const TY *Y, int n, int m, int r, double *core) {
  if (r <= 0 || m <= 0) return;
  if (n <= 0) {
    SPB_CUDA(cudaMemsetAsync(core, 0, sizeof(double) * (size_t)r * m, st));
    return;
  }
  const int colblocks = (int)cdiv(m, 128);
  // about 8 CTAs per SM in all, each chunk a multiple of the staging depth
  int chunks = std::max(1, std::min((int)cdiv(1184, colblocks), (int)cdiv(n, 4 * kCoreRows)));
  const int rows_per_chunk = (int)(cdiv(cdiv(n, chunks), kCoreRows) * kCoreRows);
  chunks = (int)cdiv(n, rows_per_chunk);
  Scratch part(sizeof(double) * (size_t)chunks * kCoreRB * m, st);
  for (int q0 = 0; q0 < r; q0 += kCoreRB) {
    core_partial_kernel<TY><<<dim3(colblocks, chunks), 128, 0, st>>>(U, Y, n, m, r, q0, rows_per_chunk,
                                                                     part.as<double>());
    SPB_LAUNCH_CHECK();
    core_reduce_kernel<<<cdiv((long long)kCoreRB * m, 256), 256, 0, st>>>(part.as<double>(), chunks, m, r, q0,
                                                                          core);
    SPB_LAUNCH_CHECK();
  }
}

void core_from_f32(cudaStream_t st, const double *U, const float *Y, int n, int m, int r, double *core) {
  core_from<float>(st, U, Y, n, m, r, core);
}
void core_from_f64(cudaStream_t st, const double *U, const double *Y, int n, int m, int r, double *core) {
  core_from<double>(st, U, Y, n, m, r, core);
}

template <typename T>
void weighted_sq(cudaStream_t st, const T *X, const T *Y, const double *w, int rows, int cols,
                 double *d_out2) {
  Scratch part(sizeof(double) * 2 * kRedBlocks, st);
  wsq_partial_kernel<T><<<kRedBlocks, 256, 0, st>>>(X, Y, w, rows, cols, part.as<double>());
  SPB_LAUNCH_CHECK();
  sum_pairs_kernel<<<1, 256, 0, st>>>(part.as<double>(), kRedBlocks, d_out2);
  SPB_LAUNCH_CHECK();
}
template void weighted_sq<double>(cudaStream_t, const double *, const double *, const double *,
                                  int, int, double *);
template void weighted_sq<float>(cudaStream_t, const float *, const float *, const double *, int,
                                 int, double *);

void householder_q(cudaStream_t st, double *A, int rows, int cols) {
  Scratch tau(sizeof(double) * cols, st), Q(sizeof(double) * (size_t)rows * cols, st);
  householder_kernel<<<1, 1024, 0, st>>>(A, rows, cols, tau.as<double>(), Q.as<double>());
  SPB_LAUNCH_CHECK();
  SPB_CUDA(cudaMemcpyAsync(A, Q.p, sizeof(double) * (size_t)rows * cols, cudaMemcpyDeviceToDevice, st));
}

// Time of the FP64 column Gram in us (within 15% over 1,536 to 80,000 rows and 320 to
// 2,002 columns): gram_f64 takes 0.2 us a row and wave, the 64-wide tiles of
// gemm 4e6 FMAs a us.
static double f64_gram_us(const double *A, int rows, int cols) {
  if (gram_f64_takes(cols, A, cols)) {
    const GramSplits g = gram_splits(cols, rows);
    return 25.0 + 0.2 * (double)g.kchunk * (double)g.waves;
  }
  const double nt = cdiv(cols, 64);
  return 30.0 + nt * (nt + 1) / 2 * 4096.0 * rows / 4e6;
}

void gram_cols(cudaStream_t st, const double *A, int rows, int cols, double *C, GramUse use) {
  if (gram::i8_gram_takes(rows, cols) && gram::i8_gram_us(rows, cols) <= f64_gram_us(A, rows, cols) &&
      gram::gram_cols_i8(st, A, rows, cols, cols, C, cols, use == GramUse::kEntries))
    return;
  gemm<double>(st, cols, cols, rows, 1.0, A, cols, true, A, cols, false, 0.0, C, cols, nullptr, true);
}

// CholQR2 calls that fell back to Householder QR (reported by the trace)
static int g_householder_fallbacks = 0;

// With dstat (2 ints on the device): the two pivot statuses go there, nothing is
// waited for, and an unsafe pivot leaves A to be thrown away by the caller.
static bool orthonormalize(cudaStream_t st, double *A, int rows, int cols, int *dstat);

bool orthonormalize(cudaStream_t st, double *A, int rows, int cols) { return orthonormalize(st, A, rows, cols, nullptr); }

static bool orthonormalize(cudaStream_t st, double *A, int rows, int cols, int *dstat) {
  if (cols > 64 || rows < cols) {
    householder_q(st, A, rows, cols);
    return true;
  }
  Scratch G(sizeof(double) * cols * cols, st), Ri(sizeof(double) * cols * cols, st),
      tmp(sizeof(double) * (size_t)rows * cols, st), stat(sizeof(int) * 2, st),
      orig(dstat ? 0 : sizeof(double) * (size_t)rows * cols, st);
  int *pstat = dstat ? dstat : stat.as<int>();
  if (!dstat)
    SPB_CUDA(cudaMemcpyAsync(orig.p, A, sizeof(double) * (size_t)rows * cols, cudaMemcpyDeviceToDevice, st));
  int hstat[2] = {0, 0};
  for (int pass = 0; pass < 2; ++pass) {
    gemm<double>(st, cols, cols, rows, 1.0, A, cols, true, A, cols, false, 0.0, G.as<double>(), cols,
                 nullptr, true);
    if (cols <= 16)
      chol_inv_warp_kernel<16><<<1, 32, 0, st>>>(G.as<double>(), cols, Ri.as<double>(), pstat + pass);
    else if (cols <= 32)
      chol_inv_warp_kernel<32><<<1, 32, 0, st>>>(G.as<double>(), cols, Ri.as<double>(), pstat + pass);
    else
      chol_inv_kernel<<<1, 256, 2 * sizeof(double) * cols * cols, st>>>(G.as<double>(), cols, Ri.as<double>(),
                                                                       pstat + pass);
    SPB_LAUNCH_CHECK();
    gemm<double>(st, rows, cols, cols, 1.0, A, cols, false, Ri.as<double>(), cols, false, 0.0,
                 tmp.as<double>(), cols);
    SPB_CUDA(cudaMemcpyAsync(A, tmp.p, sizeof(double) * (size_t)rows * cols,
                             cudaMemcpyDeviceToDevice, st));
  }
  if (dstat) return false;
  SPB_CUDA(cudaMemcpyAsync(hstat, stat.p, sizeof(int) * 2, cudaMemcpyDeviceToHost, st));
  SPB_CUDA(cudaStreamSynchronize(st));
  if (hstat[0] || hstat[1]) {
    ++g_householder_fallbacks;
    // Gram matrix numerically singular: restart from the original columns
    // with Householder QR, which is stable for any conditioning.
    SPB_CUDA(cudaMemcpyAsync(A, orig.p, sizeof(double) * (size_t)rows * cols, cudaMemcpyDeviceToDevice, st));
    householder_q(st, A, rows, cols);
    return true;
  }
  return false;
}

// W -= Q (Q^T W) twice (classical Gram-Schmidt with re-orthogonalisation)
static void project_out(cudaStream_t st, const double *Q, int ldq, int width, double *W, int s, int b,
                        double *C) {
  if (width <= 0) return;
  for (int pass = 0; pass < 2; ++pass) {
    gemm<double>(st, width, b, s, 1.0, Q, ldq, true, W, b, false, 0.0, C, b);
    gemm<double>(st, s, b, width, -1.0, Q, ldq, false, C, b, false, 1.0, W, b);
  }
}

void jacobi_eig(cudaStream_t st, const double *S, int n, double *w, double *V) {
  if (n > kJacobiMax) fail(SYMPROP_ERR_SIZE, "jacobi_eig: n=%d > %d", n, kJacobiMax);
  const int np = (n + 1) & ~1, half = np / 2, blocks = half * (half + 1) / 2;
  const size_t smem = sizeof(double) * np * (np + 1);
  Scratch rot(sizeof(double2) * (size_t)kJacobiSweeps * std::max(np - 1, 1) * half, st),
      meta(sizeof(int) * (n + 1), st);
  int *place = meta.as<int>(), *sweeps = place + n;
  SPB_CUDA(cudaFuncSetAttribute(jacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // one block of A per thread where 1024 threads can, else two
  const int threads = std::min(1024, std::max(64, (int)cdiv(blocks > 1024 ? cdiv(blocks, 2) : blocks, 32) * 32));
  jacobi_kernel<<<1, threads, smem, st>>>(S, n, w, rot.as<double2>(), place, sweeps);
  SPB_LAUNCH_CHECK();
  jacobi_vectors_kernel<<<n, 32, 0, st>>>(rot.as<double2>(), place, sweeps, n, V);
  SPB_LAUNCH_CHECK();
}

void scale_sym(cudaStream_t st, double *G, int m, const double *sd) {
  scale_sym_kernel<<<cdiv((long long)m * m, 256), 256, 0, st>>>(G, m, sd);
  SPB_LAUNCH_CHECK();
}

void scale_rows_clip(cudaStream_t st, double *U, int n, int r, double delta) {
  clip_rows_kernel<<<cdiv(n, 256), 256, 0, st>>>(U, n, r, delta);
  SPB_LAUNCH_CHECK();
}

template <typename Ts, typename Td> void convert(cudaStream_t st, const Ts *src, Td *dst, size_t n) {
  if (!n) return;
  convert_kernel<Ts, Td><<<cdiv((long long)n, 256), 256, 0, st>>>(src, dst, n);
  SPB_LAUNCH_CHECK();
}
template void convert<double, float>(cudaStream_t, const double *, float *, size_t);
template void convert<float, double>(cudaStream_t, const float *, double *, size_t);

// SPB_TRACE_EIG=1 prints the restart count and final residual of each solve
static bool eig_trace() {
  static const bool on = [] {
    const char *e = std::getenv("SPB_TRACE_EIG");
    return e && *e && *e != '0';
  }();
  return on;
}

// Block Krylov (block Lanczos with full re-orthogonalisation and thick
// restart) for the top-r eigenpairs of S.  Projected problems of at most
// kJacobiMax columns are solved by jacobi_eig.
static int top_eigs_op(cudaStream_t st, const SymApply &apply, int s, int r, double *V, double *lam,
                       const double *warm, double tol, int max_restarts, const double *dense);

int top_eigs(cudaStream_t st, const double *S, int s, int r, double *V, double *lam,
             const double *warm, double tol, int max_restarts) {
  SymApply apply = [S, s](cudaStream_t stream, const double *X, int ldx, int cols, double *Y, int ldy) {
    gemm<double>(stream, s, cols, s, 1.0, S, s, false, X, ldx, false, 0.0, Y, ldy);
  };
  return top_eigs_op(st, apply, s, r, V, lam, warm, tol, max_restarts, S);
}

int top_eigs_op(cudaStream_t st, const SymApply &apply, int s, int r, double *V, double *lam,
                const double *warm, double tol, int max_restarts) {
  return top_eigs_op(st, apply, s, r, V, lam, warm, tol, max_restarts, nullptr);
}

// dense: the matrix itself when it is at hand (small s goes straight to Jacobi)
static int top_eigs_op(cudaStream_t st, const SymApply &apply, int s, int r, double *V, double *lam,
                const double *warm, double tol, int max_restarts, const double *dense) {
  if (r > s) fail(SYMPROP_ERR_INVALID, "rank %d exceeds matrix size %d", r, s);
  if (s <= kJacobiMax) {
    Scratch w(sizeof(double) * s, st), Z(sizeof(double) * s * s, st), Sd(dense ? 0 : sizeof(double) * s * s, st);
    if (!dense) {  // form the small matrix: S = S I
      Scratch I(sizeof(double) * s * s, st);
      SPB_CUDA(cudaMemsetAsync(I.p, 0, sizeof(double) * s * s, st));
      eye_kernel<<<cdiv(s, 256), 256, 0, st>>>(I.as<double>(), s);
      SPB_LAUNCH_CHECK();
      apply(st, I.as<double>(), s, s, Sd.as<double>(), s);
      dense = Sd.as<double>();
    }
    jacobi_eig(st, dense, s, w.as<double>(), Z.as<double>());
    copy_cols_kernel<<<cdiv((long long)s * r, 256), 256, 0, st>>>(Z.as<double>(), s, s, r, V, r);
    SPB_LAUNCH_CHECK();
    SPB_CUDA(cudaMemcpyAsync(lam, w.p, sizeof(double) * r, cudaMemcpyDeviceToHost, st));
    SPB_CUDA(cudaStreamSynchronize(st));
    return SYMPROP_OK;
  }
  const int b = std::min(std::max(r + 8, 2 * r), std::min(48, s));
  if (b < r) fail(SYMPROP_ERR_SIZE, "rank %d too large for the eigensolver", r);
  // Krylov basis width: the Rayleigh-Ritz Jacobi costs O(nb^3) per restart
  // whatever s is, the products with S O(s^2 nb): small matrices take 64
  // columns, large ones the full 96 (fewer restarts); at least two blocks
  const int krylov_cols = s < 1024 ? 64 : kJacobiMax;
  const int nblk = std::max(2, krylov_cols / b);
  const int nb = nblk * b;  // Krylov basis width
  Scratch Q(sizeof(double) * (size_t)s * nb, st), SQ(sizeof(double) * (size_t)s * nb, st),
      T(sizeof(double) * nb * nb, st), w(sizeof(double) * nb, st), Z(sizeof(double) * nb * nb, st),
      C(sizeof(double) * nb * b, st), X(sizeof(double) * (size_t)s * b, st),
      SX(sizeof(double) * (size_t)s * b, st), res(sizeof(double) * b, st),
      blk(sizeof(double) * (size_t)s * b, st);
  double *q = Q.as<double>(), *sq = SQ.as<double>();
  // start block: warm subspace padded with pseudo-random columns
  random_fill_kernel<<<cdiv((long long)s * b, 256), 256, 0, st>>>(X.as<double>(), (size_t)s * b,
                                                                   0x5EED5EEDull);
  SPB_LAUNCH_CHECK();
  if (warm) {
    copy_cols_kernel<<<cdiv((long long)s * r, 256), 256, 0, st>>>(warm, r, s, r, X.as<double>(), b);
    SPB_LAUNCH_CHECK();
  }
  std::vector<double> hw(nb), hres(b);
  Scratch stat(sizeof(int) * 2 * nblk, st), X2(sizeof(double) * (size_t)s * b, st);
  std::vector<int> hstat(2 * nblk);
  double *x = X.as<double>(), *xn = X2.as<double>();
  // One restart from the block x: Krylov basis, Rayleigh-Ritz, the new block
  // in xn.  The quick form checks no pivot until the restart's only wait; when
  // one was not safe, the restart is done again in the careful form, which
  // waits for each block and falls back to Householder, and so are the
  // solve's other restarts.
  auto restart = [&](bool careful) {
    auto orth = [&](double *W, int j) {
      return orthonormalize(st, W, s, b, careful ? nullptr : stat.as<int>() + 2 * j);
    };
    if (!careful) SPB_CUDA(cudaMemsetAsync(stat.p, 0, sizeof(int) * 2 * nblk, st));
    // Q[:, 0:b] = orth(X)
    copy_cols_kernel<<<cdiv((long long)s * b, 256), 256, 0, st>>>(x, b, s, b, blk.as<double>(), b);
    SPB_LAUNCH_CHECK();
    orth(blk.as<double>(), 0);
    copy_cols_kernel<<<cdiv((long long)s * b, 256), 256, 0, st>>>(blk.as<double>(), b, s, b, q, nb);
    SPB_LAUNCH_CHECK();
    int width = b;
    for (int j = 1; j < nblk; ++j) {
      // W = S * Q[:, (j-1)b : jb], orthogonalised against the basis so far
      // (column-scaled CholQR2; Householder when W is numerically rank
      // deficient, then a second projection removes any direction it
      // invented inside the existing basis).
      apply(st, q + (j - 1) * b, nb, b, sq + (j - 1) * b, nb);
      copy_cols_kernel<<<cdiv((long long)s * b, 256), 256, 0, st>>>(sq + (j - 1) * b, nb, s, b, blk.as<double>(), b);
      SPB_LAUNCH_CHECK();
      project_out(st, q, nb, width, blk.as<double>(), s, b, C.as<double>());
      if (orth(blk.as<double>(), j)) {
        project_out(st, q, nb, width, blk.as<double>(), s, b, C.as<double>());
        householder_q(st, blk.as<double>(), s, b);
      }
      copy_cols_kernel<<<cdiv((long long)s * b, 256), 256, 0, st>>>(blk.as<double>(), b, s, b,
                                                                    q + j * b, nb);
      SPB_LAUNCH_CHECK();
      width += b;
    }
    // Rayleigh-Ritz: T = Q^T S Q (S Q of the other blocks is there)
    apply(st, q + (nblk - 1) * b, nb, b, sq + (nblk - 1) * b, nb);
    gemm<double>(st, nb, nb, s, 1.0, q, nb, true, sq, nb, false, 0.0, T.as<double>(), nb);
    jacobi_eig(st, T.as<double>(), nb, w.as<double>(), Z.as<double>());
    // X = Q Z[:, :b], SX = SQ Z[:, :b]
    copy_cols_kernel<<<cdiv((long long)nb * b, 256), 256, 0, st>>>(Z.as<double>(), nb, nb, b,
                                                                   C.as<double>(), b);
    SPB_LAUNCH_CHECK();
    gemm<double>(st, s, b, nb, 1.0, q, nb, false, C.as<double>(), b, false, 0.0, xn, b);
    gemm<double>(st, s, b, nb, 1.0, sq, nb, false, C.as<double>(), b, false, 0.0, SX.as<double>(), b);
    residual_kernel<<<r, 256, 0, st>>>(SX.as<double>(), xn, s, b, r, w.as<double>(), res.as<double>());
    SPB_LAUNCH_CHECK();
    SPB_CUDA(cudaMemcpyAsync(hw.data(), w.p, sizeof(double) * nb, cudaMemcpyDeviceToHost, st));
    SPB_CUDA(cudaMemcpyAsync(hres.data(), res.p, sizeof(double) * r, cudaMemcpyDeviceToHost, st));
    if (!careful)
      SPB_CUDA(cudaMemcpyAsync(hstat.data(), stat.p, sizeof(int) * 2 * nblk, cudaMemcpyDeviceToHost, st));
    SPB_CUDA(cudaStreamSynchronize(st));
    return careful || (std::all_of(hstat.begin(), hstat.end(), [](int v) { return v == 0; }) &&
                       !debug_value(SYMPROP_DEBUG_UNSAFE_PIVOTS));
  };
  int repeated = 0;  // restarts done twice
  bool careful = false;
  for (int it = 0; it <= max_restarts; ++it) {
    if (!careful && !restart(false)) {
      careful = true;
      ++repeated;
    }
    if (careful) restart(true);
    std::swap(x, xn);
    double scale = std::max(std::fabs(hw[0]), 1e-300);
    double worst = 0;
    for (int i = 0; i < r; ++i) worst = std::max(worst, hres[i] / scale);
    if (worst <= tol || it == max_restarts) {
      if (eig_trace())
        std::fprintf(stderr, "top_eigs: s=%d r=%d b=%d restarts=%d repeated=%d residual=%.3e tol=%.1e householder=%d\n",
                     s, r, b, it, repeated, worst, tol, g_householder_fallbacks);
      g_householder_fallbacks = 0;
      copy_cols_kernel<<<cdiv((long long)s * r, 256), 256, 0, st>>>(x, b, s, r, V, r);
      SPB_LAUNCH_CHECK();
      for (int i = 0; i < r; ++i) lam[i] = hw[i];
      SPB_CUDA(cudaStreamSynchronize(st));
      return worst <= tol ? SYMPROP_OK : SYMPROP_ERR_NOCONV;
    }
  }
  return SYMPROP_ERR_NOCONV;
}

}  // namespace dense

// Stream-ordered scratch from a pool private to this library, one per
// device, that keeps its memory between calls: the eigensolver's many small
// buffers cost no allocation after the first iteration.  What it keeps is bounded
// by two buffers of the largest size that goes there.  (The device's default pool releases
// memory at every synchronisation unless its owner raised the threshold.)
// symprop_trim_memory gives the unused part back, and so does a device buffer
// whose allocation fails.
cudaMemPool_t device_pool() {
  static std::mutex mu;
  static std::map<int, cudaMemPool_t> pools;
  int dev = 0;
  SPB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  auto it = pools.find(dev);
  if (it != pools.end()) return it->second;
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool;
  SPB_CUDA(cudaMemPoolCreate(&pool, &props));
  uint64_t keep = 2 * PoolBuf::kPoolMax;
  SPB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
  pools[dev] = pool;
  return pool;
}

void trim_pool() {
  SPB_CUDA(cudaDeviceSynchronize());
  SPB_CUDA(cudaMemPoolTrimTo(device_pool(), 0));
}

}  // namespace spb
