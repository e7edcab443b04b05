// S3TTMc, split-leaf schedule (s3ttmc_split.cu).
#pragma once

#include "tensor.cuh"

namespace spb {

// Whether the split-leaf schedule covers this order and rank.
bool split_supported(uint32_t order, uint32_t R);
// How many of the items (heaviest first) it takes at rank R; the rest are the
// warp-per-row kernel's.
uint32_t split_heavy(uint32_t R, const ItemSet &items);
// Index tables of one rank, on the device.
std::shared_ptr<SplitPlan> split_plan(uint32_t order, uint32_t R);
// One pass over the work items: packed Y rows, partial rows for split rows.
void split_launch(const SplitPlan &pl, const TensorState &t, const ItemSet &items, const void *dU, void *dYpacked,
                  int precision, cudaStream_t st);

}  // namespace spb
