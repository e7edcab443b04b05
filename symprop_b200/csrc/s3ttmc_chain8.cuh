// S3TTMc, pivot-chain schedule, order 4 at R <= 8 (s3ttmc_chain8.cu).
#pragma once

#include "s3ttmc_chain.cuh"

namespace spb {

bool chain8_supported(const TensorState &t, uint32_t R);
// chain_launch for what chain8_supported covers; items not empty.
void chain8_launch(const TensorState &t, const ChainData &cd, const ItemSet &items, const void *dU, uint32_t R,
                   void *dYpacked, int precision, cudaStream_t st);

}  // namespace spb
