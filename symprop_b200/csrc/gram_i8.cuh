// FP64 Gram on the 8-bit integer tensor cores (gram_i8.cu).
#pragma once

#include "common.cuh"

namespace spb {
namespace gram {

// Whether the column Gram of a rows x cols FP64 matrix goes to the integer
// tensor cores.
bool i8_gram_pays(int rows, int cols);
// C (cols x cols, full symmetric, row stride ldc) = A^T A for a row-major
// rows x cols FP64 A (row stride lda).  False, with C untouched, when A holds
// an infinity or a NaN, or when there is no device memory for the operands (at
// most about 4.5 GB, from the library's pool).  Waits for `st`.
bool gram_cols_i8(cudaStream_t st, const double *A, int rows, int cols, int lda, double *C, int ldc);

}  // namespace gram
}  // namespace spb
