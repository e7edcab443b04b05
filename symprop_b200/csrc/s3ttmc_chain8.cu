// S3TTMc, pivot-chain schedule at order 4, R <= 8: one warp per work item, the
// sums as products on the FP64 tensor cores (mma m8n8k4).
//
// The decomposition is that of the 128-thread kernel in s3ttmc_chain.cu (same
// owners, order, flags and items): with a row's owners sorted by (s_1, s_2),
//     W = sum c U[s_3] per prefix (s_1, s_2),
//     Q = sum U[s_2] W^T + W U[s_2]^T per group s_1,
//     G = sum U[s_1] (x) Q  (8 x 36),   Y[i] = Sym3(G).
// At R <= 8 a batch of that kernel is too little work for 128 threads: its eight
// barriers and scans per batch bound it (3.09 ms FP64 and 2.83 ms FP32 on the
// Zipf(1.1) order-4 tensor of 5,000,000 entries and 100,000 nodes at R = 8, of
// which the FMAs are 0.2 ms).  Here every sum is a product one 8-wide tile wide
// that a warp forms by itself without a barrier:
//   W  (coefficients, prefix x owner) times the owners' s_3 rows, k = owners;
//   Q  the s_2 rows times the W rows, k = prefixes; two groups at a time, because
//      a group has 1 to 4 prefixes and its products wait for one another;
//   G  the s_1 rows times the packed Q, k = groups, 4 at a time, in 10 registers.
// An owner's record is loaded two batches of 32 ahead and its s_3 row copied one
// batch ahead; the pivots' rows are copied during the W stage.  The bound is the
// latency of these steps at the 15 warps per SM that shared memory (FP64, 14 KB
// each) and registers (FP32) leave.  Measured against the 128-thread kernel, in
// ms (FP64 / FP32):
//   nodes, entries (Zipf)      R     before           now
//   100,000, 5,000,000  1.1    8     3.09 / 2.83      1.16 / 1.09
//   30,011, 900,001     1.1    8     0.621 / 0.556    0.265 / 0.256
//   30,011, 900,001     1.1    4     0.598 / 0.531    0.253 / 0.248
//   10,000, 200,000 planted    8     0.127 / 0.114    0.070 / 0.065
//   1,000, 20,000       1.2    8     0.040 / 0.037    0.025 / 0.025
// For R > 8 the same kernel with 16-wide tiles takes 236 registers, 8 warps per
// SM, and stays latency-bound: 1.1 times as fast as the 128-thread kernel on the
// largest tensor of the table and 0.75 times on the smallest, so that the
// 128-thread kernel keeps those ranks.
#include <map>
#include <mutex>

#include "s3ttmc_chain8.cuh"
#include "s3ttmc_mma.cuh"

namespace spb {
namespace {

constexpr int kR = 8, kTiles = 5;  // G: 8 x 36 in column tiles of 8
constexpr int kW = 12, kQ = 44;                 // row strides (doubles): 12 (mod 16), no bank conflicts in the
                                                // 8-byte fragment loads (8 rows of 4 lanes)
constexpr int kLdG = 41;                        // odd: column reads of G
template <typename T> constexpr int kU = sizeof(T) == 8 ? 12 : 8;
template <typename T> constexpr size_t smem_bytes() {
  return sizeof(double) * (32 * kW + 4 * kQ + 4 * kW) + sizeof(T) * 3 * 32 * kU<T> + sizeof(uint32_t) * 96;
}
static_assert(sizeof(double) * kR * kLdG <= smem_bytes<float>(), "G overlays the batch");

struct Params {
  const Chunk *chunks;
  const uint32_t *S;     // nown x 4: leaf ids in pivot order, one unused
  const void *c;         // coefficients (T)
  const uint8_t *flags;  // bit 0: starts a group, bit 1: a prefix
  const void *U;         // nrows x R (T)
  uint32_t R, m3;
  void *Y;               // packed rows (T), row stride m3
  double *partials;      // nslots x m3
  const uint2 *trip;     // m3: offsets in G of the three terms (o0 | o1 << 16, o2)
  uint64_t nown;
  uint32_t nrows, nslots;
};

__device__ __forceinline__ uint32_t shared_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Rows of U (ids in shared memory) to shared rows of stride kU, asynchronously,
// in `pieces` 16-byte pieces a row where every row of U starts on 16 bytes, else
// (pieces 0) value by value.  (A third way, 8-byte pieces, made R = 8 slower by 8%.)
template <typename T>
__device__ __forceinline__ void copy_rows(T *dst, const uint32_t *ids, int count, const T *U, int R, int pieces,
                                          int lane) {
  if (pieces) {
    constexpr int P = kR * (int)sizeof(T) / 16, E = 16 / (int)sizeof(T);
#pragma unroll 4
    for (int e = lane; e < count * P; e += 32) {
      const int h = e / P, k = e % P;
      if (k < pieces)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(shared_addr(dst + h * kU<T> + k * E)),
                     "l"(U + (uint64_t)ids[h] * R + k * E)
                     : "memory");
    }
  } else {
#pragma unroll 4
    for (int e = lane; e < count * kR; e += 32) {
      const int h = e / kR, x = e % kR;
      if (x < R)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(shared_addr(dst + h * kU<T> + x)),
                     "l"(U + (uint64_t)ids[h] * R + x), "n"((int)sizeof(T))
                     : "memory");
    }
  }
}

template <typename T> __global__ void __launch_bounds__(32, 16) s3ttmc_chain8_kernel(const Params p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *sW = reinterpret_cast<double *>(smem_raw);  // W of the batch's prefixes
  double *sQ = sW + 32 * kW;                          // Q of up to four groups
  double *sV = sQ + 4 * kQ;                           // and their s_1 rows
  T *sU2 = reinterpret_cast<T *>(sV + 4 * kW);        // s_2 rows of the prefixes
  T *sU1 = sU2 + 32 * kU<T>;                          // s_1 rows of the groups
  T *sU3 = sU1 + 32 * kU<T>;                          // s_3 rows of the owners
  uint32_t *sId3 = reinterpret_cast<uint32_t *>(sU3 + 32 * kU<T>), *sId2 = sId3 + 32, *sId1 = sId2 + 32;
  const int lane = threadIdx.x, kq = lane & 3, r8 = lane >> 2;
  const Chunk ch = p.chunks[blockIdx.x];
  if (!SPB_BOUND(ch.ob <= ch.oe && ch.oe <= p.nown && ch.row < p.nrows && (ch.slot == kDirect || ch.slot < p.nslots),
                 201, blockIdx.x))
    return;
  const T *U = reinterpret_cast<const T *>(p.U);
  const T *cc = reinterpret_cast<const T *>(p.c);
  const int R = (int)p.R;
  const int bytes = R * (int)sizeof(T),
            pieces = (bytes & 15) == 0 && (reinterpret_cast<uintptr_t>(p.U) & 15u) == 0 ? bytes / 16 : 0;
  for (int e = lane; e < 3 * 32 * kU<T>; e += 32) sU2[e] = T(0);  // columns R .. 7 stay zero
  for (int e = lane; e < 4 * kQ; e += 32) sQ[e] = 0.0;            // columns 36 .. 39 stay zero

  double g[kTiles][2];  // G: row r8, columns 8 j + 2 kq + {0, 1}
#pragma unroll
  for (int j = 0; j < kTiles; ++j) g[j][0] = g[j][1] = 0.0;
  // places of this lane's entries of a Q (row r8, columns 2 kq + {0, 1}) in the
  // packed row, -1 below the diagonal
  int qat[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int x = r8, y = 2 * kq + e;
    qat[e] = x <= y ? x * kR - (x * (x - 1)) / 2 + (y - x) : -1;
  }

  // lane l holds owner l of a batch of 32 (loaded two batches ahead of its
  // products; its s_3 row is copied one batch ahead)
  struct Rec {
    uint4 id = {0, 0, 0, 0};
    T c = T(0);
    uint32_t f = 0;
  };
  auto load_rec = [&](uint64_t o0) {
    Rec r;
    const uint64_t o = o0 + (uint64_t)lane;
    if (o < ch.oe) {
      r.id = *reinterpret_cast<const uint4 *>(p.S + o * 4);
      if (!SPB_BOUND(r.id.x < p.nrows && r.id.y < p.nrows && r.id.z < p.nrows, 202, o)) r.id = make_uint4(0, 0, 0, 0);
      r.c = cc[o];
      r.f = p.flags[o];
    }
    return r;
  };
  auto copy_u3 = [&](const Rec &r, uint64_t o0) {
    const int nb = o0 < ch.oe ? (int)min((uint64_t)32, ch.oe - o0) : 0;
    sId3[lane] = r.id.z;
    __syncwarp();
    copy_rows(sU3, sId3, nb, U, R, pieces, lane);
  };
  int slots = 0;  // groups in sQ
  // G += U[s_1] (x) Q over the groups in sQ
  auto add_groups = [&]() {
    __syncwarp();
    const double a = kq < slots ? sV[kq * kW + r8] : 0.0;
#pragma unroll
    for (int j = 0; j < kTiles; ++j) mma_f64(g[j], a, kq < slots ? sQ[kq * kQ + 8 * j + r8] : 0.0);
    __syncwarp();
    slots = 0;
  };

  Rec cur = load_rec(ch.ob), rec = load_rec(ch.ob + 32);
  __syncwarp();
  copy_u3(cur, ch.ob);
  for (uint64_t o0 = ch.ob; o0 < ch.oe; o0 += 32) {
    const int nb = (int)min((uint64_t)32, ch.oe - o0);
    const bool in = lane < nb;
    // bit l: owner l starts a group (s_1), a prefix (s_1, s_2)
    const uint32_t gm = __ballot_sync(0xffffffffu, in && (lane == 0 || (cur.f & 1u))),
                   pm = __ballot_sync(0xffffffffu, in && (lane == 0 || (cur.f & 2u)));
    const uint32_t upto = (2u << lane) - 1u;  // lanes up to this one
    const int pid = __popc(pm & upto) - 1, np = __popc(pm), ng = __popc(gm);
    if (pm >> lane & 1u) sId2[pid] = cur.id.y;
    if (gm >> lane & 1u) sId1[__popc(gm & upto) - 1] = cur.id.x;
    __syncwarp();
    // the pivots' rows, in flight during the W stage (the s_3 rows came before)
    asm volatile("cp.async.commit_group;" ::: "memory");
    copy_rows(sU2, sId2, np, U, R, pieces, lane);
    copy_rows(sU1, sId1, ng, U, R, pieces, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    // ---- W of every prefix: the matrix of coefficients (prefix x owner) times
    // the s_3 rows.  The prefixes grow along the owners, so four owners touch one
    // or two tiles of 8 prefixes.  A row with an infinity or a NaN takes the
    // plain sums (0 times it is not 0).
    T u3[8];
    bool odd = false;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      u3[k] = 4 * k + kq < nb ? sU3[(4 * k + kq) * kU<T> + r8] : T(0);
      odd = odd || !isfinite(u3[k]);
    }
    double ck[8];
    int pk[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      pk[k] = __shfl_sync(0xffffffffu, in ? pid : -1, 4 * k + kq);
      ck[k] = (double)__shfl_sync(0xffffffffu, cur.c, 4 * k + kq);
    }
    if (!__any_sync(0xffffffffu, odd)) {
      double w[2][2] = {{0.0, 0.0}, {0.0, 0.0}};  // even and odd steps apart: two chains of products
      int tile = 0;
      auto flush = [&]() {
        *reinterpret_cast<double2 *>(&sW[(8 * tile + r8) * kW + 2 * kq]) =
            make_double2(w[0][0] + w[1][0], w[0][1] + w[1][1]);
        w[0][0] = w[0][1] = w[1][0] = w[1][1] = 0.0;
      };
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (4 * k >= nb) break;
        // tiles of the prefixes of owners 4 k and 4 k + 3 (owners past the batch start none)
        const int t0 = (__popc(pm & ((2u << (4 * k)) - 1u)) - 1) >> 3,
                  t1 = (__popc(pm & ((16u << (4 * k)) - 1u)) - 1) >> 3;
        if (t0 != tile) {
          flush();
          tile = t0;
        }
        mma_f64(w[k & 1], pk[k] == 8 * tile + r8 ? ck[k] : 0.0, (double)u3[k]);
        if (t1 != tile) {
          flush();
          tile = t1;
          mma_f64(w[k & 1], pk[k] == 8 * tile + r8 ? ck[k] : 0.0, (double)u3[k]);
        }
      }
      flush();
    } else {
      for (int e = lane; e < 32 * kW; e += 32) sW[e] = 0.0;
      __syncwarp();
      for (int k = 0; k < nb; ++k) {
        const int q = __shfl_sync(0xffffffffu, pid, k);
        const T c = __shfl_sync(0xffffffffu, cur.c, k);
        if (lane < R) sW[q * kW + lane] += (double)c * (double)sU3[k * kU<T> + lane];
        __syncwarp();
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    // the next batch's s_3 rows, in flight during the rest
    cur = rec;
    copy_u3(cur, o0 + 32);
    rec = load_rec(o0 + 64);
    // ---- Q of every group: sum over its prefixes of U2 W^T + W U2^T; two
    // groups at a time (their chains of products are short)
    int p1 = 0, gi = 0;  // prefixes and groups done
    for (uint32_t left = gm & (gm - 1u); gi < ng;) {
      // group gi: prefixes [pa, pb), group gi + 1: [pb, pc)
      const int pa = p1, pb = left ? __popc(pm & ((left & (0u - left)) - 1u)) : np;
      left &= left - 1u;
      const bool two = gi + 1 < ng;
      const int pc = !two ? pb : left ? __popc(pm & ((left & (0u - left)) - 1u)) : np;
      left &= left - 1u;
      p1 = pc;
      double q[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      const int steps = max(pb - pa, pc - pb);
      for (int h0 = 0; h0 < steps; h0 += 4) {
        double u[2], v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int h = (i ? pb : pa) + h0 + kq;
          const bool on = h < (i ? pc : pb);
          u[i] = on ? (double)sU2[h * kU<T> + r8] : 0.0;
          v[i] = on ? sW[h * kW + r8] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_f64(q[i], u[i], v[i]);
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_f64(q[i], v[i], u[i]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (i && !two) break;
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (qat[e] >= 0) sQ[slots * kQ + qat[e]] = q[i][e];
        if (lane < kR) sV[slots * kW + lane] = (double)sU1[(gi + i) * kU<T> + lane];
        if (++slots == 4) add_groups();
      }
      gi += 2;
    }
    __syncwarp();  // before the next batch's rows
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (slots) add_groups();
  // ---- Y = Sym3(G) through shared memory
  __syncwarp();
  double *sG = reinterpret_cast<double *>(smem_raw);  // 8 rows of stride kLdG
#pragma unroll
  for (int j = 0; j < kTiles; ++j) {
    sG[r8 * kLdG + 8 * j + 2 * kq] = g[j][0];
    sG[r8 * kLdG + 8 * j + 2 * kq + 1] = g[j][1];
  }
  __syncwarp();
#pragma unroll 4
  for (uint32_t e = lane; e < p.m3; e += 32) {
    const uint2 o = p.trip[e];
    const double y = sG[o.x & 0xffffu] + sG[o.x >> 16] + sG[o.y];
    if (ch.slot == kDirect) reinterpret_cast<T *>(p.Y)[(uint64_t)ch.row * p.m3 + e] = (T)y;
    else p.partials[(uint64_t)ch.slot * p.m3 + e] = y;
  }
}

// offsets in G (rows of stride kLdG, pairs packed for 8 columns) of the three
// terms of every packed entry of rank R
const uint2 *triples8(uint32_t R) {
  static std::mutex mu;
  // kept for the life of the process (at most 1 KB per rank and device)
  static std::map<std::pair<int, uint32_t>, uint2 *> cache;
  int dev = 0;
  SPB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  uint2 *&slot = cache[{dev, R}];
  if (!slot) {
    auto at = [](uint32_t row, uint32_t x, uint32_t y) { return row * kLdG + x * kR - x * (x - 1) / 2 + (y - x); };
    std::vector<uint2> h;
    for_each_sorted(R, 3, [&](const std::vector<uint32_t> &q, uint64_t) {
      h.push_back(make_uint2(at(q[0], q[1], q[2]) | at(q[1], q[0], q[2]) << 16, at(q[2], q[0], q[1])));
    });
    uint2 *d = nullptr;
    SPB_CUDA(cudaMalloc(&d, h.size() * sizeof(uint2)));
    SPB_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(uint2), cudaMemcpyHostToDevice));
    slot = d;
  }
  return slot;
}

template <typename T> void go(const Params &p, uint32_t nchunks, cudaStream_t st) {
  s3ttmc_chain8_kernel<T><<<nchunks, 32, smem_bytes<T>(), st>>>(p);
  SPB_LAUNCH_CHECK();
}

}  // namespace

bool chain8_supported(const TensorState &t, uint32_t R) {
  return t.order == 4 && t.sstride == 4 && R >= 1 && R <= (uint32_t)kR;
}

void chain8_launch(const TensorState &t, const ChainData &cd, const ItemSet &items, const void *dU, uint32_t R,
                   void *dYpacked, int precision, cudaStream_t st) {
  Params p;
  p.chunks = items.chunks;
  p.S = cd.S;
  p.c = precision == SYMPROP_FP64 ? (const void *)cd.c64 : (const void *)cd.c32;
  p.flags = cd.flags;
  p.U = dU;
  p.R = R;
  p.m3 = (uint32_t)symsize(R, 3);
  p.Y = dYpacked;
  p.partials = items.partials;
  p.trip = triples8(R);
  p.nown = t.nown;
  p.nrows = t.dim;
  p.nslots = items.nslots;
  if (precision == SYMPROP_FP64) go<double>(p, items.nchunks, st);
  else go<float>(p, items.nchunks, st);
  spb_check_host(st, "S3TTMc chain kernel (R <= 8)");
}

}  // namespace spb
