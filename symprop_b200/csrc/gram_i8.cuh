// FP64 Gram on the 8-bit integer tensor cores (gram_i8.cu).
#pragma once

#include "common.cuh"

namespace spb {
namespace gram {

// Whether gram_cols_i8 is for the column Gram of a rows x cols FP64 matrix, and about
// how long it takes (us).
bool i8_gram_takes(int rows, int cols);
double i8_gram_us(int rows, int cols);
// C (cols x cols, full symmetric, row stride ldc) = A^T A for a row-major
// rows x cols FP64 A (row stride lda), each entry within about 2^-53 |a_i| |a_j|
// (columns of A).  componentwise: within rows * 2^-53 sum_k |a_ki| |a_kj| as well,
// the bound of a sum in FP64.  False when A holds an infinity
// or a NaN, when a componentwise Gram has many columns whose large entries lie
// in different rows, or when the device has no memory for the operands of
// about 1,000 rows.  Of the operands the library's pool keeps at most 4.5 GB.  Waits for `st`,
// except for the last sums of odd entries.
bool gram_cols_i8(cudaStream_t st, const double *A, int rows, int cols, int lda, double *C, int ldc,
                  bool componentwise);

}  // namespace gram
}  // namespace spb
