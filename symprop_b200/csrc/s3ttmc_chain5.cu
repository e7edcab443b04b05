// S3TTMc, pivot-chain schedule for order 5, group kernel: the owners of a row
// grouped by their first pivot, the groups multiplied on the FP64 tensor cores.
//
// A leaf S = {s_1, ..., s_4} in pivot order (s3ttmc_chain.cu) has the tensor
// (the reference's SymOuterProd recursion,
// include/detail/dense/symtensor.hpp:24-39, src/compressed_dtree.cpp:421-518)
//     K(S)[q] = sum_t U[s_1][q_t] P3(s_2, s_3, s_4)[q without q_t],
//     P3[x y z] = the sum over the 6 orderings of U[s_2][.] U[s_3][.] U[s_4][.],
// so a row is
//     Y[i] = Sym4(G),  G = sum_g U[s_1(g)] (x) T_g          (R x m3, m3 = R(R+1)(R+2)/6)
//     T_g = sum over the owners of g of c P3
//     Sym4(G)[q] = sum_t G[q_t][q without q_t].
// The owners of a row are sorted by pivots, so a group is a run of owners with
// the same s_1, cut into sub-groups of at most 16 owners.  G is a matrix
// product whose inner dimension is the sub-groups (13,056 FMAs each at
// R = 16), T_g a sum in registers (2,448 FMAs and 816 for the pair products
// per owner).  On the order-5 power-law workload there are 0.19 groups per
// owner.
//
// One persistent CTA per SM: 8 warps hold G (8 x 8 tiles, every warp all row
// tiles and every eighth column tile) and multiply stages of 8 sub-groups, 8
// warps build them, one sub-group each: lane and set give a pair (x <= y) of
// places, the entries (x, y, z >= y) of T are the lane's registers, and the
// columns z of the leaf's U rows come from shared memory, the same for all
// lanes.  Within an item the sub-groups are ordered by size, so that the 8 of a
// stage take the same time.  Two stages, handed over with named barriers; the
// 4 terms per entry of an item are added by the multiplying warps while the
// builders work on the next one.  FP32 builds T in FP32 (paired FMAs) and
// widens it in the multipliers; G is summed in FP64 either way.
//
// Bounds: at R <= 8 the latency of a stage (two CTAs an SM hide part of it); above,
// the building warps: 3,264 FMAs per owner at R = 16 at 8 warps an SM, beside the FP64
// tensor instructions, which hold the FP64 pipe.  The CTA-per-item kernel of
// s3ttmc_chain.cu (chain5_rows_launch) forms F = U[s_2] (x) T3 per prefix instead and
// passes every batch through five barriers.  Measured against it, in ms:
//   order 5, nodes, tuples              R     FP64 before, now   FP32 before, now
//   20,000, 2,000,000 power-law        16     13.2   (12.9)      6.82   5.41
//                                      12     13.4    6.00       6.71   3.68
//                                       8     12.3    3.35       6.23   2.05
//   5,000, 200,000 Zipf(1.1)           16      1.33  (1.62)      0.710  0.698
//                                       9      1.09   0.696      0.557  0.436
//   100,000, 200,000 Zipf(1.1)         16      5.91  (7.00)      3.34  (3.85)
//                                      12      4.33   2.90       2.39  (2.55)
//                                       7      3.05   1.21       1.62   0.944
//   250, 10,000 Zipf(1.2)               8      0.061  0.044      0.055  0.030
// (in brackets: measured, not chosen).  The rule (chain5_pays): FP64 at R > 12
// stays with the CTA kernel, T and G taking more registers than there are (70 and
// 104 a thread of 128); FP32 at R > 8 comes here where a node has 64 owners on
// average, because closing an item (all of G through shared memory) costs as much
// as some tens of owners (at 25 owners a node the two are equal, at 10 this one
// takes 1.15 times as long, at 200 it is the faster one), and at R > 12 only with at
// least one group (s_1) to 10 owners: the CTA kernel gains from owners that share
// pivots, this one hardly.  FP32, R = 16, ms, CTA kernel / this one, by groups an owner:
//   1,000 nodes, 200,000 equal degrees    0.43    1.778  0.980
//   20,000, 2,000,000 power-law           0.19    6.82   5.41
//   20,000, 300,000 Zipf(1.05)            0.155   1.693  1.446
//   3,000, 60,000 Zipf(1.1)               0.103   0.272  0.271
//   10,000, 400,000 Zipf(1.1)             0.078   1.344  1.346
//   1,000, 20,000 Zipf(1.2)               0.069   0.095  0.104
//   1,000, 50,000 Zipf(1.2)               0.043   0.156  0.177
//   3,000, 600,000 Zipf(1.1)              0.035   1.307  1.460
// (R = 12 on the last one: 1.331 / 0.980.)
//
// The first call on a tensor also orders its owners (chain_data: two radix sorts)
// and deals them to the warps (chain5_build); both are kept.  First call, ms, FP32,
// before this kernel / now: 250 nodes, 10,000 tuples, R = 8 1.02 / 0.67; 10,000 nodes,
// 200,000 tuples 8.6 / 1.7; 20,000 nodes, 2M tuples, R = 16 16.7 / 10.3; 200,000 nodes,
// 20M tuples 127 / 95.
#include <cub/cub.cuh>

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "s3ttmc_chain.cuh"
#include "s3ttmc_mma.cuh"

namespace spb {
namespace {

constexpr int kMulWarps = 8, kBuildWarps = 8, kMul = 32 * kMulWarps, kBuild = 32 * kBuildWarps;
constexpr int kThreads = kMul + kBuild;
constexpr int kK = kBuildWarps;  // sub-groups per stage
constexpr int kSub = 16;         // owners per sub-group
template <typename T> constexpr int kBlk = sizeof(T) == 8 ? 2 : 4;  // owners gathered at a time by a warp
constexpr int kStages = 2;
constexpr uint32_t kLast = 0x80000000u;
constexpr int kFirst = kBuildWarps + 1;  // places of an item in `first`

// Places of T: by the middle index y, then z, then x (the lanes of a set, pairs
// with the same y next to each other, store next to each other).
// y of the first pair of set s (pairs by y, then x, 32 to a set); an
// expression, so that the unrolled loops see a constant
__host__ __device__ constexpr int low_of(int s) { return s == 0 ? 0 : s == 1 ? 7 : s == 2 ? 10 : s == 3 ? 13 : 15; }

// y of its last pair
__host__ __device__ constexpr int high_of(int s) { return s == 0 ? 7 : s == 1 ? 10 : s == 2 ? 13 : 15; }

// asynchronous copy of one value, global -> shared
__device__ __forceinline__ void copy_async(double *d, const double *g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(g) : "memory");
}
__device__ __forceinline__ void copy_async(float *d, const float *g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(g) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int RZ, typename T> struct Geo5 {
  static constexpr int pairs = RZ * (RZ + 1) / 2, elems = RZ * (RZ + 1) * (RZ + 2) / 6;
  static constexpr int NS = (pairs + 31) / 32;         // pair sets
  static constexpr int MT = (RZ + 7) / 8;              // row tiles of G
  static constexpr int n8 = (elems + 7) / 8;           // column tiles
  static constexpr int NT = (n8 + kMulWarps - 1) / kMulWarps;
  static constexpr int sA = 8 * MT + 4;                // doubles; 4 or 12 (mod 16): conflict-free fragment loads
  static constexpr int pad_b() {
    int s = 8 * n8;
    if (sizeof(T) == 8) return s + 4;                  // 4 or 12 (mod 16) doubles
    while (s % 32 != 8 && s % 32 != 24) s += 8;        // 8 or 24 (mod 32) floats
    return s;
  }
  static constexpr int sB = pad_b();
  static constexpr int ldG = 8 * n8 + 1;
  static constexpr int leaf = 4 * RZ;                  // staged leaf: rows s_2, s_3, c s_4, s_1
};

struct GroupParams {
  const Chunk *chunks;  // ob: number of the item in row order, oe - ob: its sub-groups
  uint32_t nchunks;
  const uint32_t *first;  // 9 per item: the first owner of each building warp, the end of the last's
  const uint32_t *S;      // nown x 4 leaf ids in pivot order; kLast in s_1 of a sub-group's last owner
  const double *c;
  const void *U;
  uint32_t R, m;
  void *Y;
  double *partials;
  const uint16_t *quad;   // m: q0 | q1 << 4 | q2 << 8 | q3 << 12 of an entry
  uint64_t nentries, nown;
  uint32_t nrows, nslots;
};

enum { kBarFull = 1, kBarEmpty = kBarFull + kStages, kBarMul = kBarEmpty + kStages };

template <int RZ, typename T> constexpr size_t group5_smem() {
  using G = Geo5<RZ, T>;
  return sizeof(double) * kStages * kK * G::sA +
         sizeof(T) * (kStages * kK * G::sB + 8 * G::MT * G::ldG + kBuildWarps * 2 * kBlk<T> * G::leaf) +
         sizeof(uint32_t) * (kBuildWarps * 8 + 2 * RZ) + sizeof(uint16_t) * (RZ * (RZ + 1) * (RZ + 2) * (RZ + 3) / 24 + 1);
}

template <int RZ, int CTAS, typename T>
__global__ void __launch_bounds__(kThreads, CTAS) s3ttmc_group5_kernel(const GroupParams p) {
  using G = Geo5<RZ, T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *sA = reinterpret_cast<double *>(smem_raw);          // kStages x kK x sA: the s_1 rows
  T *sB = reinterpret_cast<T *>(sA + kStages * kK * G::sA);   // kStages x kK x sB: T of every sub-group
  T *sUall = sB + kStages * kK * G::sB;                       // kBuildWarps x 2 blocks of staged leaves
  T *sG = sUall + kBuildWarps * 2 * kBlk<T> * G::leaf;        // 8 MT x ldG
  uint32_t *sState = reinterpret_cast<uint32_t *>(sG + 8 * G::MT * G::ldG);  // kBuildWarps x 8
  // entry (x, y, z) of T is at place sF[y].x + z sF[y].y + x
  int2 *sF = reinterpret_cast<int2 *>(sState + 8 * kBuildWarps);
  uint16_t *sQuad = reinterpret_cast<uint16_t *>(sF + RZ);    // m entries
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint32_t e = tid; e < p.m; e += kThreads) sQuad[e] = p.quad[e];
  if (tid < RZ) {
    int o = -tid * (tid + 1);
    for (int k = 0; k < tid; ++k) o += (RZ - k) * (k + 1);
    sF[tid] = make_int2(o, tid + 1);
  }
  __syncthreads();

  if (warp < kMulWarps) {
    const int kq = lane & 3, r8 = lane >> 2;
    const int nn = (G::n8 - warp + kMulWarps - 1) / kMulWarps;
    double acc[G::NT][G::MT][2];
#pragma unroll
    for (int j = 0; j < G::NT; ++j)
#pragma unroll
      for (int i = 0; i < G::MT; ++i) acc[j][i][0] = acc[j][i][1] = 0.0;
    auto none = [](uint32_t, uint32_t) {};
    Walk<kK> w;
    w.start(p);
    w.open(p, none);
    for (int n = 0; w.valid(p); ++n) {
      const int s = n % kStages;
      const int steps = (w.count() + 3) >> 2;
      bar_sync<kThreads>(kBarFull + s);
      for (int k = 0; k < steps; ++k) {
        const double *A = sA + (s * kK + 4 * k + kq) * G::sA + r8;
        const T *B = sB + (s * kK + 4 * k + kq) * G::sB + 8 * warp + r8;
        double a[G::MT];
#pragma unroll
        for (int i = 0; i < G::MT; ++i) a[i] = A[8 * i];
#pragma unroll
        for (int j = 0; j < G::NT; ++j) {
          if (j >= nn) break;
          const double b = (double)B[8 * kMulWarps * j];
#pragma unroll
          for (int i = 0; i < G::MT; ++i) mma_f64(acc[j][i], a[i], b);
        }
      }
      bar_arrive<kThreads>(kBarEmpty + s);
      if (w.last()) {
        // the item's G through shared memory, then the 4 terms of its entries;
        // the building warps go on with the next item meanwhile
#pragma unroll
        for (int j = 0; j < G::NT; ++j)
#pragma unroll
          for (int i = 0; i < G::MT; ++i) {
            if (j < nn) {
              T *d = sG + (8 * i + r8) * G::ldG + 8 * (warp + kMulWarps * j) + 2 * kq;
              d[0] = (T)acc[j][i][0];
              d[1] = (T)acc[j][i][1];
            }
            acc[j][i][0] = acc[j][i][1] = 0.0;
          }
        bar_sync<kMul>(kBarMul);
#pragma unroll 4
        for (uint32_t e = tid; e < p.m; e += kMul) {
          const uint32_t q = sQuad[e];
          const int q0 = q & 15, q1 = (q >> 4) & 15, q2 = (q >> 8) & 15, q3 = q >> 12;
          const int2 f1 = sF[q1], f2 = sF[q2];
          const int z1 = f1.x + q0, z2 = f2.x + q3 * f2.y;
          const double y = (double)sG[q0 * G::ldG + z2 + q1] + (double)sG[q1 * G::ldG + z2 + q0] +
                           (double)sG[q2 * G::ldG + z1 + q3 * f1.y] + (double)sG[q3 * G::ldG + z1 + q2 * f1.y];
          put<T>(p, w.row, w.slot, e, y);
        }
        bar_sync<kMul>(kBarMul);
      }
      w.next(p, none);
    }
    return;
  }

  // ---- building warps
  constexpr int kB = kBlk<T>;
  const int bt = tid - kMul, bw = warp - kMulWarps;
  const T *U = reinterpret_cast<const T *>(p.U);
  T *sU = sUall + bw * 2 * kB * G::leaf;
  for (int e = lane; e < 2 * kB * G::leaf; e += 32) sU[e] = T(0);  // columns R .. RZ - 1 stay zero
  // items of this CTA: sub-groups, and this warp's owners [q, end)
  struct Item {
    uint32_t subs = 0, q = 0, end = 0;
  };
  auto item_at = [&](uint32_t i) {
    Item r;
    if (i < p.nchunks) {
      const Chunk ch = p.chunks[i];
      if (SPB_BOUND(ch.ob <= ch.oe && ch.oe <= p.nentries && ch.row < p.nrows &&
                        (ch.slot == kDirect || ch.slot < p.nslots),
                    511, i)) {
        r.subs = (uint32_t)(ch.oe - ch.ob);
        if (r.subs) {
          r.q = p.first[ch.ob * kFirst + bw];
          r.end = p.first[ch.ob * kFirst + bw + 1];
          if (!SPB_BOUND(r.q <= r.end && r.end <= p.nown, 512, r.q)) r.q = r.end = 0;
        }
      }
    }
    return r;
  };
  // The warp's owners, item after item in the order they are stored, in blocks
  // of kB (a block ends with its item): the ids of a block are loaded two
  // blocks ahead, its U rows copied to shared memory one block ahead.
  // The state that only changes between blocks lives in shared memory (the
  // registers are T's): the next block starts at f_q of item f_item.
  enum { kFItem, kFQ, kFEnd, kNextQ, kNextEnd, kSubs1, kQ1, kEnd1 };
  volatile uint32_t *state = sState + 8 * bw;
  struct Block {
    int count = 0;
    uint32_t id = 0;  // lane 4 i + k: id k of owner i
    double c = 0.0;   // lane i: coefficient of owner i (rounded to T where it is used: a
                      // conversion here would wait for the load)
  };
  auto next_ids = [&](Block &r) {
    uint32_t f_q = state[kFQ], f_end = state[kFEnd], f_item = state[kFItem];
    while (f_q == f_end && f_item < p.nchunks) {  // warp-uniform
      f_item += gridDim.x;
      f_q = state[kNextQ];
      f_end = state[kNextEnd];
      const Item x = item_at(f_item + gridDim.x);
      __syncwarp();
      state[kFItem] = f_item;
      state[kFEnd] = f_end;
      state[kNextQ] = x.q;
      state[kNextEnd] = x.end;
      __syncwarp();
    }
    r.count = (int)min((uint32_t)kB, f_end - f_q);
    r.id = 0;
    r.c = 0.0;
    if (lane < 4 * r.count) {
      r.id = p.S[(uint64_t)f_q * 4 + lane];
      if (!SPB_BOUND((r.id & ~kLast) < p.nrows, 513, f_q)) r.id &= kLast;
    }
    if (lane < r.count) r.c = p.c[f_q + lane];
    __syncwarp();
    state[kFQ] = f_q + (uint32_t)r.count;
    __syncwarp();
  };
  const int x0 = lane & 15, half = lane >> 4;
  auto copy_rows = [&](const Block &b, int buf) {
#pragma unroll
    for (int i = 0; i < kB; ++i) {
      const uint32_t i23 = __shfl_sync(0xffffffffu, b.id, 4 * i + 1 + half),
                     i41 = __shfl_sync(0xffffffffu, b.id, 4 * i + (half ? 0 : 3)) & ~kLast;
      if (i < b.count && x0 < (int)p.R) {
        T *u = sU + (buf * kB + i) * G::leaf + half * RZ + x0;
        copy_async(u, U + (uint64_t)i23 * p.R + x0);
        copy_async(u + 2 * RZ, U + (uint64_t)i41 * p.R + x0);
      }
    }
  };
  // this lane's pairs: set s holds pairs 32 s + lane in order of y, then x
  // (packed x | y << 8 | d0 << 16; entry (x, y, z) goes to place d0 + z (y + 1))
  int pr[G::NS];
#pragma unroll
  for (int s = 0; s < G::NS; ++s) {
    const int e = min(32 * s + lane, G::pairs - 1);
    int y = 0;
    while ((y + 1) * (y + 2) / 2 <= e) ++y;
    const int x = e - y * (y + 1) / 2;
    int d0 = x - y * (y + 1);
    for (int k = 0; k < y; ++k) d0 += (RZ - k) * (k + 1);
    pr[s] = x | y << 8 | d0 << 16;
  }
  T acc[G::NS][RZ];  // entries (px, py, z) of T; z below the set's first y unused
#pragma unroll
  for (int s = 0; s < G::NS; ++s)
#pragma unroll
    for (int z = 0; z < RZ; ++z) acc[s][z] = T(0);
  int n = 0;  // stages so far
  // hands over this warp's place of the next stage, which has `places` of them:
  // T and the s_1 row (in u), or zeros that pad the last step
  auto emit = [&](int places, const T *u) {
    const int s = n % kStages;
    if (n >= kStages) bar_sync<kThreads>(kBarEmpty + s);
    if (bw < ((places + 3) & ~3)) {
      T *B = sB + (s * kK + bw) * G::sB;
      double *A = sA + (s * kK + bw) * G::sA;
#pragma unroll
      for (int t = 0; t < G::NS; ++t) {
        const bool has = 32 * t + 31 < G::pairs || 32 * t + lane < G::pairs;
        const int y = (pr[t] >> 8) & 0xff;
        T *d = B + (pr[t] >> 16);
#pragma unroll
        for (int z = low_of(t); z < RZ; ++z) {
          if (has && (z >= high_of(t) || z >= y)) d[z * (y + 1)] = acc[t][z];
          acc[t][z] = T(0);
        }
      }
      if constexpr (G::elems % 8 != 0)
        if (lane < 8 * G::n8 - G::elems) B[G::elems + lane] = T(0);
      if (lane < 8 * G::MT) A[lane] = u && lane < RZ ? (double)u[3 * RZ + lane] : 0.0;
    }
    bar_arrive<kThreads>(kBarFull + s);
    ++n;
  };

  Item it = item_at(blockIdx.x);  // the item being built; the next one in state[kSubs1 ..]
  {
    const Item x = item_at(blockIdx.x + gridDim.x);
    state[kFItem] = blockIdx.x;
    state[kFQ] = it.q;
    state[kFEnd] = it.end;
    state[kNextQ] = state[kQ1] = x.q;
    state[kNextEnd] = state[kEnd1] = x.end;
    state[kSubs1] = x.subs;
  }
  __syncwarp();
  Block nxt, fut;  // being copied, ids being loaded
  next_ids(nxt);
  int buf = 0;
  copy_rows(nxt, buf);
  next_ids(fut);
  for (uint32_t i = blockIdx.x; i < p.nchunks; i += gridDim.x) {
    if (!it.subs) {  // a row without owners
      const Chunk ch = p.chunks[i];
      if (SPB_BOUND(ch.row < p.nrows && (ch.slot == kDirect || ch.slot < p.nslots), 514, i))
        for (uint32_t e = bt; e < p.m; e += kBuild) put<T>(p, ch.row, ch.slot, e, 0.0);
    }
    int left = (int)it.subs;  // sub-groups from the next stage on
#pragma unroll 1
    for (uint32_t q = it.q; q < it.end; q += kB) {
      copy_wait();
      __syncwarp();  // nxt's rows have arrived, and all lanes are done with the other buffer
      const int count = nxt.count;
      const uint32_t id = nxt.id;
      // the coefficients go with the s_4 rows
      const T cs = (T)nxt.c;
#pragma unroll
      for (int e = 0; e < kB * 16; e += 32) {
        const int o = (e >> 4) + half;
        const T c = __shfl_sync(0xffffffffu, cs, o);
        if (x0 < (int)p.R) sU[(buf * kB + o) * G::leaf + 2 * RZ + x0] *= c;
      }
      copy_rows(fut, buf ^ 1);
      nxt = fut;
      next_ids(fut);
      __syncwarp();
#pragma unroll 1
      for (int o = 0; o < count; ++o) {
        const T *u = sU + (buf * kB + o) * G::leaf;
        if constexpr (sizeof(T) == 8) {
#pragma unroll
          for (int t = 0; t < G::NS; ++t) {
            const T *ux = u + (pr[t] & 0xff), *uy = u + ((pr[t] >> 8) & 0xff);
            const T a0 = ux[0], a1 = ux[RZ], a2 = ux[2 * RZ], b0 = uy[0], b1 = uy[RZ], b2 = uy[2 * RZ];
            const T p01 = a0 * b1 + a1 * b0, p02 = a0 * b2 + a2 * b0, p12 = a1 * b2 + a2 * b1;
#pragma unroll
            for (int z = low_of(t) & ~1; z < RZ; z += 2) {
              const double2 z0 = *reinterpret_cast<const double2 *>(u + z),
                            z1 = *reinterpret_cast<const double2 *>(u + RZ + z),
                            z2 = *reinterpret_cast<const double2 *>(u + 2 * RZ + z);
              if (z >= low_of(t)) acc[t][z] = fma(p01, z2.x, fma(p02, z1.x, fma(p12, z0.x, acc[t][z])));
              acc[t][z + 1] = fma(p01, z2.y, fma(p02, z1.y, fma(p12, z0.y, acc[t][z + 1])));
            }
          }
        } else {
          T p01[G::NS], p02[G::NS], p12[G::NS];
#pragma unroll
          for (int t = 0; t < G::NS; ++t) {
            const T *ux = u + (pr[t] & 0xff), *uy = u + ((pr[t] >> 8) & 0xff);
            const T a0 = ux[0], a1 = ux[RZ], a2 = ux[2 * RZ], b0 = uy[0], b1 = uy[RZ], b2 = uy[2 * RZ];
            p01[t] = a0 * b1 + a1 * b0, p02[t] = a0 * b2 + a2 * b0, p12[t] = a1 * b2 + a2 * b1;
          }
#pragma unroll
          for (int z = 0; z < RZ; z += 4) {
            const float4 z0 = *reinterpret_cast<const float4 *>(u + z),
                         z1 = *reinterpret_cast<const float4 *>(u + RZ + z),
                         z2 = *reinterpret_cast<const float4 *>(u + 2 * RZ + z);
#pragma unroll
            for (int t = 0; t < G::NS; ++t) {
              if (z + 1 >= low_of(t)) {
                fma2(acc[t][z], acc[t][z + 1], p01[t], z2.x, z2.y);
                fma2(acc[t][z], acc[t][z + 1], p02[t], z1.x, z1.y);
                fma2(acc[t][z], acc[t][z + 1], p12[t], z0.x, z0.y);
              }
              if (z + 3 >= low_of(t)) {
                fma2(acc[t][z + 2], acc[t][z + 3], p01[t], z2.z, z2.w);
                fma2(acc[t][z + 2], acc[t][z + 3], p02[t], z1.z, z1.w);
                fma2(acc[t][z + 2], acc[t][z + 3], p12[t], z0.z, z0.w);
              }
            }
          }
        }
        if (__shfl_sync(0xffffffffu, id, 4 * o) & kLast) {
          emit(left, u);
          left -= kK;
        }
      }
      buf ^= 1;
    }
    for (; left > 0; left -= kK) emit(left, nullptr);  // stages in which this warp has no sub-group
    it.subs = state[kSubs1];
    it.q = state[kQ1];
    it.end = state[kEnd1];
    const Item x = item_at(i + 2 * gridDim.x);
    __syncwarp();
    state[kSubs1] = x.subs;
    state[kQ1] = x.q;
    state[kEnd1] = x.end;
    __syncwarp();
  }
  copy_wait();
  for (int s = 0; s < min(n, kStages); ++s) bar_sync<kThreads>(kBarEmpty + s);
}

// Sub-groups of one item (at most 1024 owners; S in pivot order): owner i starts one when it
// starts a group (flag bit 0, or the item's first owner) or is a multiple of
// kSub owners into its group.  Their number goes to count[item].  They are dealt to
// the building warps by size, largest first (sub-group r of that stable order to
// warp r % 8, stage r / 8), and the owners stored warp by warp in that order:
// S_out[k], c_out[k] are those of place k, kLast set where it ends its sub-group,
// first[9 item + w] is warp w's first place (w = 8: the item's end).
// The order is worked out in shared memory, so that the copies run along places.
__global__ void __launch_bounds__(128) sub_groups_kernel(const Chunk *items, const uint8_t *flags, uint32_t *count,
                                                         const uint4 *S, const double *c, uint4 *S_out, double *c_out,
                                                         uint32_t *first) {
  constexpr int kPer = 8;
  using Scan = cub::BlockScan<int, 128>;
  using Sort = cub::BlockRadixSort<uint32_t, 128, kPer, uint32_t>;
  __shared__ union {
    typename Scan::TempStorage scan;
    typename Sort::TempStorage sort;
  } tmp;
  __shared__ uint16_t starts[128 * kPer + 1];
  __shared__ uint32_t sub[128 * kPer];     // by size: start | owners << 16
  __shared__ uint16_t place[128 * kPer];   // first place of the sub-group among its warp's
  __shared__ uint16_t from[128 * kPer];    // owner of each place, bit 15: ends its sub-group
  __shared__ uint32_t wsum[kBuildWarps];
  const Chunk ch = items[blockIdx.x];
  const int n = (int)(ch.oe - ch.ob), t = threadIdx.x;
  int head[kPer], prev = 0;  // the group start at or before owner i (of this thread so far)
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = t * kPer + j;
    if (i < n && (i == 0 || (flags[ch.ob + i] & 1))) prev = i;
    head[j] = prev;
  }
  int before;
  Scan(tmp.scan).ExclusiveScan(prev, before, 0, cub::Max());
  __syncthreads();
  bool st[kPer];
  int cnt = 0, rank, total;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = t * kPer + j;
    st[j] = i < n && ((i - max(head[j], before)) & (kSub - 1)) == 0;
    cnt += st[j];
  }
  Scan(tmp.scan).ExclusiveSum(cnt, rank, total);
  if (t == 0) count[blockIdx.x] = (uint32_t)total;
#pragma unroll
  for (int j = 0; j < kPer; ++j)
    if (st[j]) starts[rank++] = (uint16_t)(t * kPer + j);
  if (t == 0) starts[total] = (uint16_t)n;
  __syncthreads();
  uint32_t key[kPer], val[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int r = t * kPer + j;
    const uint32_t b = r < total ? starts[r] : 0, len = r < total ? starts[r + 1] - b : 0;
    key[j] = kSub - len;  // the unused places last
    val[j] = b | len << 16;
  }
  Sort(tmp.sort).Sort(key, val, 0, 5);
#pragma unroll
  for (int j = 0; j < kPer; ++j) sub[t * kPer + j] = val[j];
  __syncthreads();
  if (t < kBuildWarps) {
    uint32_t o = 0;
    for (int r = t; r < total; r += kBuildWarps) {
      place[r] = (uint16_t)o;
      o += sub[r] >> 16;
    }
    wsum[t] = o;
  }
  __syncthreads();
  if (t <= kBuildWarps) {
    uint32_t o = (uint32_t)ch.ob;
    for (int w = 0; w < t; ++w) o += wsum[w];
    first[(size_t)blockIdx.x * kFirst + t] = o;
  }
  for (int r = t; r < total; r += 128) {
    const int w = r % kBuildWarps;
    uint32_t o = place[r];
    for (int k = 0; k < w; ++k) o += wsum[k];
    const uint32_t b = sub[r] & 0xffffu, len = sub[r] >> 16;
    for (uint32_t j = 0; j < len; ++j) from[o + j] = (uint16_t)((b + j) | (j + 1 == len ? 0x8000u : 0u));
  }
  __syncthreads();
  for (int k = t; k < n; k += 128) {
    const uint32_t f = from[k], i = f & 0x7fffu;
    uint4 v = S[ch.ob + i];
    if (f & 0x8000u) v.x |= kLast;
    S_out[ch.ob + k] = v;
    c_out[ch.ob + k] = c[ch.ob + i];
  }
}

constexpr int rank_size(uint32_t R) { return R <= 8 ? 8 : R <= 12 ? 12 : 16; }

// The ids of every packed entry of rank R (kept per device and rank for the
// life of the process, at most 8 KB each)
const uint16_t *quad_table(uint32_t R) {
  static std::mutex mu;
  static std::map<std::pair<int, uint32_t>, uint16_t *> cache;
  int dev = 0;
  SPB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  uint16_t *&slot = cache[{dev, R}];
  if (slot) return slot;
  std::vector<uint16_t> h;
  for_each_sorted(R, 4, [&](const std::vector<uint32_t> &q, uint64_t) {
    h.push_back((uint16_t)(q[0] | q[1] << 4 | q[2] << 8 | q[3] << 12));
  });
  uint16_t *d = nullptr;
  SPB_CUDA(cudaMalloc(&d, h.size() * sizeof(uint16_t)));
  SPB_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(uint16_t), cudaMemcpyHostToDevice));
  return slot = d;
}

template <int RZ, int CTAS, typename T> void go(const GroupParams &p, cudaStream_t st) {
  constexpr size_t smem = group5_smem<RZ, T>();
  static_assert(smem <= 227 * 1024 / CTAS - 1024 * (CTAS - 1), "shared memory");
  auto kern = s3ttmc_group5_kernel<RZ, CTAS, T>;
  SPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int dev = 0, nsm = 0;
  SPB_CUDA(cudaGetDevice(&dev));
  SPB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  kern<<<std::min<uint32_t>(p.nchunks, (uint32_t)(nsm * CTAS)), kThreads, smem, st>>>(p);
  SPB_LAUNCH_CHECK();
}

template <typename T> void dispatch(const GroupParams &p, cudaStream_t st) {
  switch (rank_size(p.R)) {
    case 8: go<8, 2, T>(p, st); break;
    case 12: go<12, 1, T>(p, st); break;
    default:
      if constexpr (sizeof(T) == 4) go<16, 1, T>(p, st);
      else fail(SYMPROP_ERR_SIZE, "order-5 group kernel: rank %u in FP64", p.R);
  }
}

}  // namespace

void chain5_tables(uint32_t R) { quad_table(R); }

// both sides of each line: the table above
bool chain5_pays(const TensorState &t, const ChainData &cd, uint32_t R, int precision) {
  if (t.order != 5 || !chain_supported(t, R) || t.sstride != 4) return false;
  if (precision == SYMPROP_FP64) return R <= 12;
  if (R <= 8) return true;
  return t.nown >= 64ull * t.dim && (R <= 12 || 10 * cd.ngroups >= t.nown);
}

std::unique_ptr<ChainGroups> chain5_build(const TensorState &t, const ChainData &cd, const std::vector<Chunk> &items) {
  NvtxRange nv("chain groups");
  const size_t n = items.size();
  auto g = std::make_unique<ChainGroups>();
  g->sub.assign(n, 0);
  Places pl;
  const size_t at_S = pl.add<uint32_t>(t.nown * 4), at_c = pl.add<double>(t.nown), at_f = pl.add<uint32_t>(n * kFirst);
  cudaStream_t st = 0;
  g->store.alloc(pl.bytes, st);
  g->S = reinterpret_cast<uint32_t *>(g->store.p + at_S);
  g->c = reinterpret_cast<double *>(g->store.p + at_c);
  g->first = reinterpret_cast<uint32_t *>(g->store.p + at_f);
  if (!n) return g;
  PoolBuf tmp(n * (sizeof(Chunk) + sizeof(uint32_t)), st);
  Chunk *const d = tmp.as<Chunk>();
  uint32_t *const count = reinterpret_cast<uint32_t *>(d + n);
  SPB_CUDA(cudaMemcpyAsync(d, items.data(), n * sizeof(Chunk), cudaMemcpyHostToDevice, st));
  sub_groups_kernel<<<(unsigned)n, 128, 0, st>>>(d, cd.flags, count, reinterpret_cast<const uint4 *>(cd.S),
                                                 cd.c64, reinterpret_cast<uint4 *>(g->S), g->c, g->first);
  SPB_LAUNCH_CHECK();
  SPB_CUDA(cudaMemcpyAsync(g->sub.data(), count, n * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  SPB_CUDA(cudaStreamSynchronize(st));
  return g;
}

void chain5_launch(const TensorState &t, const ChainData &cd, const ItemSet &items, const void *dU, uint32_t R,
                   void *dYpacked, int precision, cudaStream_t st) {
  GroupParams p{};
  p.chunks = items.chunks;
  p.nchunks = items.nchunks;
  p.first = cd.groups->first;
  p.S = cd.groups->S;
  p.c = cd.groups->c;
  p.U = dU;
  p.R = R;
  p.m = (uint32_t)symsize(R, 4);
  p.Y = dYpacked;
  p.partials = items.partials;
  p.quad = quad_table(R);
  p.nentries = cd.groups->sub.size() + 1024;  // item number + sub-groups
  p.nown = t.nown;
  p.nrows = t.dim;
  p.nslots = items.nslots;
  if (precision == SYMPROP_FP64) dispatch<double>(p, st);
  else dispatch<float>(p, st);
  spb_check_host(st, "S3TTMc chain kernel (order 5)");
}

}  // namespace spb
