// S3TTMc, split-leaf schedule (order 6, R <= 10): a row of Y as one matrix
// product over its owners, on the FP64 tensor cores.
//
// The reference's leaf tensor (SymOuterProd recursion,
// include/detail/dense/symtensor.hpp:24-39, src/compressed_dtree.cpp:421-518)
// of a leaf S = {s_1, ..., s_5} is the sum over the orderings of S of
// prod_k U[s_pi(k)][q_k].  Split S into A = {s_1, s_2, s_3} and
// B = {s_4, s_5}, P_A and P_B the same sums over the orderings of the parts
// (packed orders 3 and 2): then
//     K(S)[q] = sum over the 10 places I of A in q of P_A[q_I] P_B[q without I]
// and the row is
//     Y[i][q] = sum_I M[q_I][q without I],  M = sum over its owners c P_A (x) P_B.
// M (220 x 55 at R = 10) is a matrix product with the row's owners as its
// inner dimension: 12,100 FMAs per owner and about 1,100 to build P_A and
// P_B, against about 32,000 for the level recursion, and the 10 terms are
// added once per row.
//
// Bound: the FP64 tensor pipe (mma.m8n8k4.f64: 64 FMAs per SM and clock, the
// rate of the FP64 pipe, measured 36.6 TFLOP/s from 4 warps per SM on).  FP32
// runs on the same product: the panels are built in FP32 and widened when
// they are stored, M is summed in FP64 (error against 64 bits 7e-8, 2e-7 with
// the level recursion's compensated FP32 sums).  12 M owners at R = 10 (order
// 6, 2M planted tuples, n = 50,000): 196 clocks each, 8.1 ms at the full
// rate; FP32 63.1 -> 12.5 ms against the team kernel (s3ttmc_warp.cu).  On 1M
// planted tuples (120 owners a row) it is 2.1x (R = 5, FP32) to 5.1x (R = 10,
// FP32) faster than the warp and team kernels, FP64 at R = 10 45.3 -> 10.4 ms.
//
// One persistent CTA per SM (R > 6): 8 warps multiply (warp w: row tiles
// w % 4 + 4 i, column tiles w / 4 + 2 j, so that every SM sub-partition holds
// the same number of 8 x 8 tiles), 8 warps gather the U rows and build the
// panels of the next 16 owners in a ring of two stages, and add the 10 terms
// of the previous item while the multipliers work on the next one.  The
// building warps work in T: FP64 arithmetic beside the multipliers waits for
// the pipe they keep full (a 30-instruction chain took 1000 clocks), which is
// why FP32 panels are not built in FP64, why M is kept in T, and why FP64
// gains less.  Stages are handed over with named barriers.  Panel rows are 4
// (mod 16) doubles apart: the fragments' 8-byte loads are free of bank
// conflicts.
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "check.cuh"
#include "s3ttmc_mma.cuh"
#include "s3ttmc_split.cuh"

namespace spb {

struct SplitPlan {
  uint32_t R = 0, m = 0;
  DBuf<uint32_t> pairs;  // x | y << 8 of the packed order-2 places, in the kernel's order
  DBuf<uint32_t> elems;  // pair (x, y) | z << 8 of the packed order-3 places
  DBuf<uint32_t> sym;    // 5 planes of m: offsets in M of the 10 terms of an entry, two per word
};

namespace {

constexpr int kL = 5;                   // leaf size
constexpr int kTerms = 10;              // C(5, 3)
constexpr int kMulWarps = 8, kMul = kMulWarps * 32;
constexpr int kK = 16;                  // owners per stage
constexpr int kStages = 2;
// M of R = 11 has 36 x 9 tiles: 45 of a multiplying warp are 180 registers of sums
// (it has 168), and in FP64 M and the panels are 268 KB of shared memory.
constexpr int kMaxR = 10;

// Sizes of the kernel for ranks up to RZ.  Panel rows are a multiple of 32
// places long (what the lanes of a building warp write; the places beyond
// the packed sizes hold values that no entry of Y reads) plus 4 doubles.
template <int RZ> struct Geo {
  static constexpr int pairs = RZ * (RZ + 1) / 2, elems = RZ * (RZ + 1) * (RZ + 2) / 6;
  static constexpr int NP = (pairs + 31) / 32, NE = (elems + 31) / 32;  // places per lane
  static constexpr int nA8 = (elems + 7) / 8, nB8 = (pairs + 7) / 8;    // 8-wide tiles of M
  static constexpr int MT = (nA8 + 3) / 4, NT = (nB8 + 1) / 2;          // tiles per multiplying warp
  static constexpr int sA = 32 * NE + 4, sB = 32 * NP + 4, ldM = 8 * nB8 + 1;
  static constexpr int panel = kK * (sA + sB);
};

struct SplitParams {
  const Chunk *chunks;
  uint32_t nchunks;
  const uint32_t *S;
  uint32_t sstride;
  const double *c;
  const void *U;
  uint32_t R;
  void *Y;
  double *partials;
  uint32_t m, npair, nelem;
  const uint32_t *pairs, *elems, *sym;
  uint64_t nentries;  // owners
  uint32_t nrows, nslots;
};

enum { kBarFull = 1, kBarEmpty = kBarFull + kStages, kBarM = kBarEmpty + kStages, kBarMFree };

// Three shared values: one 16-byte load of a group of four (FP32), three
// 8-byte loads (FP64: groups of three fall on different banks, 16-byte loads
// of groups of four would not)
template <typename T> constexpr int kG3 = sizeof(T) == 8 ? 3 : 4;
__device__ __forceinline__ void load3(const float *p, float (&v)[3]) {
  const float4 a = *reinterpret_cast<const float4 *>(p);
  v[0] = a.x, v[1] = a.y, v[2] = a.z;
}
__device__ __forceinline__ void load3(const double *p, double (&v)[3]) { v[0] = p[0], v[1] = p[1], v[2] = p[2]; }
__device__ __forceinline__ void store3(float *p, float a, float b, float c) {
  *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, 0.f);
}
__device__ __forceinline__ void store3(double *p, double a, double b, double c) { p[0] = a, p[1] = b, p[2] = c; }
// A staged leaf: RZ groups (U[s_1][x], U[s_2][x], U[s_3][x]), then RZ groups
// (U[s_4][x], c U[s_5][x])
template <typename T, int RZ> constexpr int kLeaf = RZ * (kG3<T> + 2);

template <int RZ, int BW, typename T> constexpr size_t split_smem(bool sym_shared, uint32_t m) {
  using G = Geo<RZ>;
  return sizeof(double) * kStages * G::panel +
         sizeof(T) * (8 * G::nA8 * G::ldM + kK * kLeaf<T, RZ> + BW * 32 * G::NP * kG3<T>) + (sym_shared ? sizeof(uint32_t) * (kTerms / 2) * m : 0);
}

// RZ: the rank, rounded up to the next even size that has a kernel; BW:
// building warps; REGS: the registers of a multiplying thread when the two
// roles share them unevenly; SYM: the offsets of the 10 terms in shared memory
template <int RZ, int BW, int REGS, int CTAS, bool SYM, typename T>
__global__ void __launch_bounds__(kMul + 32 * BW, CTAS) s3ttmc_split_kernel(const SplitParams p) {
  using G = Geo<RZ>;
  constexpr int kBuild = 32 * BW, kThreads = kMul + kBuild;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *panel = reinterpret_cast<double *>(smem_raw);             // kStages x kK x (sA + sB)
  T *sUall = reinterpret_cast<T *>(panel + kStages * G::panel);     // kK staged leaves
  T *sPall = sUall + kK * kLeaf<T, RZ>;                             // BW x pairs x kG3
  T *sM = sPall + BW * 32 * G::NP * kG3<T>;                         // 8 nA8 x ldM
  uint32_t *sSym = reinterpret_cast<uint32_t *>(sM + 8 * G::nA8 * G::ldM);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kK * kLeaf<T, RZ>; i += kThreads) sUall[i] = T(0);  // columns R .. RZ - 1 stay zero
  if constexpr (SYM)
    for (uint32_t i = tid; i < kTerms / 2 * p.m; i += kThreads) sSym[i] = p.sym[i];
  __syncthreads();

  if (warp < kMulWarps) {
    if constexpr (REGS > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
    const int mg = warp & 3, ng = warp >> 2;
    const int nm = (G::nA8 - mg + 3) >> 2, nn = (G::nB8 - ng + 1) >> 1;
    const int kq = lane & 3, r8 = lane >> 2;
    double acc[G::MT][G::NT][2];
#pragma unroll
    for (int i = 0; i < G::MT; ++i)
#pragma unroll
      for (int j = 0; j < G::NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    auto none = [](uint32_t, uint32_t) {};
    Walk<kK> w;
    w.start(p);
    w.open(p, none);
    bool m_used = false;
    for (int n = 0; w.valid(p); ++n) {
      const int s = n % kStages;
      const int steps = (w.count() + 3) >> 2;
      bar_sync<kThreads>(kBarFull + s);
      const double *A = panel + s * G::panel + kq * G::sA + 8 * mg + r8;
      const double *B = panel + s * G::panel + kK * G::sA + kq * G::sB + 8 * ng + r8;
      auto step = [&](const double *A, const double *B) {
        double a[G::MT], b[G::NT];
#pragma unroll
        for (int i = 0; i < G::MT; ++i) a[i] = i < nm ? A[32 * i] : 0.0;
#pragma unroll
        for (int j = 0; j < G::NT; ++j) b[j] = j < nn ? B[16 * j] : 0.0;
#pragma unroll
        for (int j = 0; j < G::NT; ++j) {
          if (j >= nn) break;
#pragma unroll
          for (int i = 0; i < G::MT; ++i)
            if (i < nm) mma_f64(acc[i][j], a[i], b[j]);
        }
      };
      if (steps == kK / 4) {
#pragma unroll
        for (int k = 0; k < kK / 4; ++k) step(A + 4 * k * G::sA, B + 4 * k * G::sB);
      } else {
        for (int k = 0; k < steps; ++k) step(A + 4 * k * G::sA, B + 4 * k * G::sB);
      }
      bar_arrive<kThreads>(kBarEmpty + s);
      if (w.last()) {
        if (m_used) bar_sync<kThreads>(kBarMFree);
        m_used = true;
#pragma unroll
        for (int i = 0; i < G::MT; ++i)
#pragma unroll
          for (int j = 0; j < G::NT; ++j) {
            if (i < nm && j < nn) {
              T *d = sM + (8 * (mg + 4 * i) + r8) * G::ldM + 8 * (ng + 2 * j) + 2 * kq;
              d[0] = (T)acc[i][j][0];
              d[1] = (T)acc[i][j][1];
            }
            acc[i][j][0] = acc[i][j][1] = 0.0;
          }
        bar_arrive<kThreads>(kBarM);
      }
      w.next(p, none);
    }
    return;
  }

  // ---- building warps: warp bw owns the leaves OW bw .. OW bw + OW - 1 of
  // every stage; nothing but the stage itself is shared between them
  if constexpr (REGS > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(256 - REGS));
  constexpr int OW = kK / BW, kVal = (OW * kL * RZ + 31) / 32;
  const int bt = tid - kMul, bw = warp - kMulWarps;
  using V2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  const T *U = reinterpret_cast<const T *>(p.U);
  const int R = (int)p.R;
  T *sU = sUall + bw * OW * kLeaf<T, RZ>, *sP = sPall + bw * 32 * G::NP * kG3<T>;
  auto zero_row = [&](uint32_t row, uint32_t slot) {
    for (uint32_t e = bt; e < p.m; e += kBuild) put<T>(p, row, slot, e, 0.0);
  };
  // add the terms of the item that the multipliers left in M
  const uint32_t *sym = SYM ? sSym : p.sym;
  auto finish = [&](uint32_t row, uint32_t slot, bool more) {
    bar_sync<kThreads>(kBarM);
#pragma unroll 2
    for (uint32_t e = bt; e < p.m; e += kBuild) {
      T y0 = T(0), y1 = T(0);
#pragma unroll
      for (int t = 0; t < kTerms / 2; ++t) {
        const uint32_t o = sym[t * p.m + e];
        y0 += sM[o & 0xffffu];
        y1 += sM[o >> 16];
      }
      put<T>(p, row, slot, e, (double)(y0 + y1));
    }
    if (more) bar_arrive<kThreads>(kBarMFree);
  };
  // lane 5 j + k holds the id at place k of the warp's leaf j (kNone beyond
  // the batch) and the factor of that row, loaded two batches ahead; the
  // values lane + 32 q of the leaves' rows are loaded one batch ahead
  constexpr uint32_t kNone = 0xffffffffu;
  int vrow[kVal], vsrc[kVal], vdst[kVal];
#pragma unroll
  for (int q = 0; q < kVal; ++q) {
    const int e = lane + 32 * q, r = e / R;
    vrow[q] = r < OW * kL ? r : 31;  // lane 31 holds kNone
    vsrc[q] = e - r * R;
    const int k = r % kL;
    vdst[q] = r < OW * kL ? (r / kL) * kLeaf<T, RZ> + (k < 3 ? vsrc[q] * kG3<T> + k : RZ * kG3<T> + vsrc[q] * 2 + k - 3)
                          : -1;
  }
  const int own_l = lane / kL, place_l = lane - own_l * kL;
  auto load_ids = [&](const Walk<kK> &w, uint32_t &id, double &c) {
    const uint32_t o = w.o + (uint32_t)(bw * OW + own_l);
    id = kNone;
    c = 0.0;
    if (w.valid(p) && own_l < OW && o < w.oe) {
      id = p.S[(uint64_t)o * p.sstride + place_l];
      if (!SPB_BOUND(id < p.nrows, 502, id)) id = 0;
      c = place_l == kL - 1 ? p.c[o] : 1.0;
    }
  };
  auto load_vals = [&](uint32_t id, double c, T (&v)[kVal], T (&f)[kVal]) {
#pragma unroll
    for (int q = 0; q < kVal; ++q) {
      const uint32_t i = __shfl_sync(0xffffffffu, id, vrow[q]);
      f[q] = __shfl_sync(0xffffffffu, (T)c, vrow[q]);
      v[q] = i != kNone ? U[(uint64_t)i * p.R + vsrc[q]] : T(0);
    }
  };
  // this lane's places: pairs lane + 32 h and order-3 places lane + 32 i (the
  // ones beyond the packed sizes repeat the first)
  int px[G::NP], py[G::NP], ep[G::NE], ez[G::NE];
#pragma unroll
  for (int h = 0; h < G::NP; ++h) {
    const uint32_t e = (uint32_t)(lane + 32 * h), t = p.pairs[e < p.npair ? e : 0];
    px[h] = (int)(t & 0xffu);
    py[h] = (int)(t >> 8);
  }
#pragma unroll
  for (int i = 0; i < G::NE; ++i) {
    const uint32_t e = (uint32_t)(lane + 32 * i), t = p.elems[e < p.nelem ? e : 0];
    ep[i] = (int)(t & 0xffu) * kG3<T>;
    ez[i] = (int)(t >> 8) * kG3<T>;
  }
  Walk<kK> w, w1;
  w.start(p);
  w.open(p, zero_row);
  if (!w.valid(p)) return;
  T v[kVal], f[kVal];
  uint32_t id;
  double c;
  load_ids(w, id, c);
  load_vals(id, c, v, f);
  w1 = w;
  w1.next(p, zero_row);
  load_ids(w1, id, c);
  bool pend = false;
  uint32_t pend_row = 0, pend_slot = 0;
  int n = 0;
  for (; w.valid(p); ++n) {
    const int s = n % kStages, nb = w.count();
#pragma unroll
    for (int q = 0; q < kVal; ++q)
      if (vdst[q] >= 0) sU[vdst[q]] = f[q] * v[q];
    Walk<kK> w2 = w1;
    if (w1.valid(p)) {
      load_vals(id, c, v, f);
      w2.next(p, zero_row);
      load_ids(w2, id, c);
    }
    __syncwarp();
    if (n >= kStages) bar_sync<kThreads>(kBarEmpty + s);
    // the last step's places beyond the batch get zeros: their leaves are staged as zeros
    const int nb4 = (nb + 3) & ~3;
    double *A = panel + s * G::panel + lane, *B = panel + s * G::panel + kK * G::sA + lane;
#pragma unroll
    for (int j = 0; j < OW; ++j) {
      const int k = bw * OW + j;
      if (k >= nb4) break;  // warp-uniform
      const T *u = sU + j * kLeaf<T, RZ>, *ub = u + RZ * kG3<T>;
#pragma unroll
      for (int h = 0; h < G::NP; ++h) {
        T a[3], b[3];
        load3(u + px[h] * kG3<T>, a);
        load3(u + py[h] * kG3<T>, b);
        store3(sP + (lane + 32 * h) * kG3<T>, a[0] * b[1] + a[1] * b[0], a[0] * b[2] + a[2] * b[0],
               a[1] * b[2] + a[2] * b[1]);
        const V2 bx = *reinterpret_cast<const V2 *>(ub + 2 * px[h]), by = *reinterpret_cast<const V2 *>(ub + 2 * py[h]);
        B[k * G::sB + 32 * h] = (double)(bx.x * by.y + bx.y * by.x);
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < G::NE; ++i) {
        T pp[3], uz[3];
        load3(sP + ep[i], pp);
        load3(u + ez[i], uz);
        A[k * G::sA + 32 * i] = (double)(pp[0] * uz[2] + pp[1] * uz[1] + pp[2] * uz[0]);
      }
      __syncwarp();
    }
    bar_arrive<kThreads>(kBarFull + s);
    if (w.first && pend) finish(pend_row, pend_slot, true);
    if (w.first) pend = false;
    if (w.last()) {
      pend = true;
      pend_row = w.row;
      pend_slot = w.slot;
    }
    w = w1;
    w1 = w2;
  }
  finish(pend_row, pend_slot, false);
  for (int s = 0; s < min(n, kStages); ++s) bar_sync<kThreads>(kBarEmpty + s);
}

template <int RZ, int BW, int REGS, int CTAS, typename T> void go(const SplitParams &p, cudaStream_t st) {
  constexpr uint32_t mz = RZ * (RZ + 1) * (RZ + 2) * (RZ + 3) * (RZ + 4) / 120;  // packed width at rank RZ
  constexpr bool SYM = split_smem<RZ, BW, T>(true, mz) <= 227 * 1024 / CTAS - 1024;
  const size_t smem = split_smem<RZ, BW, T>(SYM, p.m);
  auto kern = s3ttmc_split_kernel<RZ, BW, REGS, CTAS, SYM, T>;
  SPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int dev = 0, nsm = 0;
  SPB_CUDA(cudaGetDevice(&dev));
  SPB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  kern<<<std::min<uint32_t>(p.nchunks, (uint32_t)(nsm * CTAS)), kMul + 32 * BW, smem, st>>>(p);
  SPB_LAUNCH_CHECK();
}

template <typename T> void dispatch(const SplitParams &p, cudaStream_t st) {
  // tiles of M per warp: 28 x 7 in all at R = 10, 15 x 5 at 8, 7 x 3 at 6, 3 x 2 at 4
  if (p.R <= 4) go<4, 4, 0, 2, T>(p, st);
  else if (p.R <= 6) go<6, 4, 0, 2, T>(p, st);
  else if (p.R <= 8) go<8, 8, 0, 1, T>(p, st);
  else go<10, 8, 168, 1, T>(p, st);
}

}  // namespace

bool split_supported(uint32_t order, uint32_t R) { return order == kL + 1 && R >= 1 && R <= (uint32_t)kMaxR; }

// A row costs the split kernel about 1,500 (R = 4) to 4,000 clocks (R = 8) of
// one CTA whatever its owners (M through shared memory, 10 terms an entry), the
// warp kernel a fixed time per owner: on rows of 1 to 3 owners the warp kernel
// is 1.2x to 2.2x faster up to R = 8, on rows of 6 the two are within 6% to
// 20% either way.  At R = 9 and 10 the warp kernel's team form (s3ttmc_warp.cu)
// is the slower one at every length.
uint32_t split_heavy(uint32_t R, const ItemSet &items) { return R <= 8 ? items.nheavy : items.nchunks; }

// The tables of a rank are kept per device for the life of the process (at most 43 KB
// each): made for every tensor they were a third of the first call on a small one (order 6,
// 4,000 tuples, R = 4, FP32).
std::shared_ptr<SplitPlan> split_plan(uint32_t order, uint32_t R) {
  if (!split_supported(order, R)) fail(SYMPROP_ERR_SIZE, "split S3TTMc does not support order %u rank %u", order, R);
  static std::mutex mu;
  static auto &plans = *new std::map<std::pair<int, uint32_t>, std::shared_ptr<SplitPlan>>;  // outlives the context
  int dev = 0;
  SPB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (const auto it = plans.find({dev, R}); it != plans.end()) return it->second;
  auto pl = std::make_shared<SplitPlan>();
  pl->R = R;
  pl->m = (uint32_t)symsize(R, kL);
  // lexicographic: consecutive lanes of a building warp share the pair and
  // read consecutive U columns, and consecutive entries of Y read M along a
  // row or a column (odd stride)
  std::vector<uint32_t> pairs, elems, at2(R * R), at3(R * R * R);
  for (uint32_t x = 0; x < R; ++x)
    for (uint32_t y = x; y < R; ++y) {
      at2[x * R + y] = (uint32_t)pairs.size();
      pairs.push_back(x | y << 8);
    }
  for (uint32_t x = 0; x < R; ++x)
    for (uint32_t y = x; y < R; ++y)
      for (uint32_t z = y; z < R; ++z) {
        at3[(x * R + y) * R + z] = (uint32_t)elems.size();
        elems.push_back(at2[x * R + y] | z << 8);
      }
  const uint32_t RZ = R <= 4 ? 4 : R <= 6 ? 6 : R <= 8 ? 8 : 10, ldM = 8 * ((RZ * (RZ + 1) / 2 + 7) / 8) + 1;
  std::vector<uint32_t> sym((size_t)kTerms / 2 * pl->m, 0);
  for_each_sorted(R, kL, [&](const std::vector<uint32_t> &q, uint64_t lin) {
    int t = 0;
    for (int a = 0; a < kL; ++a)
      for (int b = a + 1; b < kL; ++b) {  // a, b: the places of B
        uint32_t r[3];
        int c = 0;
        for (int k = 0; k < kL; ++k)
          if (k != a && k != b) r[c++] = q[k];
        const uint32_t o = at3[(r[0] * R + r[1]) * R + r[2]] * ldM + at2[q[a] * R + q[b]];
        sym[(size_t)(t / 2) * pl->m + lin] |= o << (16 * (t & 1));
        ++t;
      }
  });
  pl->elems.alloc(elems.size());
  SPB_CUDA(cudaMemcpy(pl->elems.p, elems.data(), elems.size() * 4, cudaMemcpyHostToDevice));
  pl->pairs.alloc(pairs.size());
  SPB_CUDA(cudaMemcpy(pl->pairs.p, pairs.data(), pairs.size() * 4, cudaMemcpyHostToDevice));
  pl->sym.alloc(sym.size());
  SPB_CUDA(cudaMemcpy(pl->sym.p, sym.data(), sym.size() * 4, cudaMemcpyHostToDevice));
  return plans[{dev, R}] = pl;
}

void split_launch(const SplitPlan &pl, const TensorState &t, const ItemSet &items, const void *dU, void *dYpacked,
                  int precision, cudaStream_t st) {
  if (!items.nchunks) return;
  SplitParams p{};
  p.chunks = items.chunks;
  p.nchunks = items.nchunks;
  p.S = t.own_S.p;
  p.sstride = t.sstride;
  p.c = t.own_c64.p;
  p.U = dU;
  p.R = pl.R;
  p.npair = pl.R * (pl.R + 1) / 2;
  p.nelem = (uint32_t)symsize(pl.R, 3);
  p.Y = dYpacked;
  p.partials = t.partials.p;
  p.m = pl.m;
  p.pairs = pl.pairs.p;
  p.elems = pl.elems.p;
  p.sym = pl.sym.p;
  p.nentries = t.nown;
  p.nrows = t.dim;
  p.nslots = t.nslots;
  if (precision == SYMPROP_FP64) dispatch<double>(p, st);
  else dispatch<float>(p, st);
  spb_check_host(st, "S3TTMc split kernel");
}

}  // namespace spb
