// S3TTMc, pivot-chain schedule (s3ttmc_chain.cu).
#pragma once

#include "tensor.cuh"

namespace spb {

// Work items of the chain schedule, all rows and by bands.
struct ChainItems {
  uint32_t chunk_owners = 0;
  uint32_t nchunks = 0, nsplit = 0, nslots = 0;
  DBuf<Chunk> chunks;             // work items of the heavy rows, heaviest first
  DBuf<SplitRow> split;
  uint32_t nlight = 0;            // rows of at most kChainLight owners, one item
  DBuf<Chunk> light;              // each, for the warp-per-row kernel, heaviest first
  std::map<uint32_t, std::unique_ptr<RowBands>> bands;  // by band count
  bool groups = false;            // order 5: items of s3ttmc_chain5.cu
  DBuf<double> partials;          // order 4, R <= 8: partial rows of its own (it has more slots, and a
                                  // call must not move the rows of one at R > 8, captured in a graph)
};

// Order 5: the owners of every item in the order the building warps of
// s3ttmc_chain5.cu take them.  Built on first use of a rank it covers.
struct ChainGroups {
  KeptBuf store;                  // of the arrays
  uint32_t *S = nullptr;          // nown x 4 leaf ids in pivot order; bit 31 of s_1: ends its sub-group
  double *c = nullptr;            // owner coefficients
  uint32_t *first = nullptr;      // per item in row order: the first owner of each warp, the item's end
  std::vector<uint32_t> sub;      // per item: its sub-groups
};

// Owners re-sorted for the chain schedule, built on first use.
struct ChainData {
  uint32_t L = 0;                 // leaf size (order - 1)
  KeptBuf store;                  // of the arrays
  uint32_t *S = nullptr;          // nown x sstride leaf ids, highest-degree first
  double *c64 = nullptr;          // owner coefficients in chain order
  float *c32 = nullptr;
  uint8_t *flags = nullptr;       // bit k: the owner starts a new prefix of k+1 pivots
  uint64_t ngroups = 0;           // runs of owners of a row with the same first pivot
  std::unique_ptr<ChainGroups> groups;
  bool no_groups = false;         // no memory for them: the CTA kernel runs instead
  // items, by kernel: the CTA kernels; the warp kernel (order 4, R <= 8) or the
  // group kernel (order 5)
  std::unique_ptr<ChainItems> items[2];
};

// Order 4: rows with at most this many owners share few pivots; the chain
// schedule hands them to the warp-per-row kernel.  Order 5 keeps every row
// (the team kernel costs about 9x the chain's FMAs per owner).
constexpr uint64_t kChainLight = 16;
uint64_t chain_light_max(const TensorState &t);

// Whether the chain schedule covers this tensor and rank.
bool chain_supported(const TensorState &t, uint32_t R);
// The chain data of t (built on the first call).
ChainData &chain_data(TensorState &t);
// The work items of a rank and precision (built on first use), and in nb row bands.
// While a stream is captured, when none can be built, another kernel's list does: at
// order 4 either serves both kernels, at order 5 the CTA kernel's is made together with
// the group kernel's.
ChainItems &chain_items(TensorState &t, uint32_t R, int precision, bool capturing = false);
const ChainItems *built_chain_items(const TensorState &t, uint32_t R);  // null before the first use
const RowBands &chain_bands(TensorState &t, ChainItems &items, uint32_t nb);
// One pass over chain work items: packed Y rows, partial rows for split rows.
void chain_launch(const TensorState &t, const ChainData &cd, const ItemSet &items, const void *dU, uint32_t R,
                  void *dYpacked, int precision, cudaStream_t st);

// s3ttmc_chain5.cu (order 5): whether the group kernel is the faster one here;
// the owners of items (ranges in row order of the owners in pivot order), dealt to
// its warps; one pass over items whose ob is the item's number in row order and
// whose oe - ob is its number of sub-groups.
bool chain5_pays(const TensorState &t, const ChainData &cd, uint32_t R, int precision);
void chain5_tables(uint32_t R);  // its index table of a rank, built on first use
std::unique_ptr<ChainGroups> chain5_build(const TensorState &t, const ChainData &cd, const std::vector<Chunk> &items);
void chain5_launch(const TensorState &t, const ChainData &cd, const ItemSet &items, const void *dU, uint32_t R,
                   void *dYpacked, int precision, cudaStream_t st);

}  // namespace spb
