// Sizes of the pieces in which the fast-diagonalisation passes stage their
// operands; plain host and device arithmetic.
#pragma once
#include <cuda_runtime.h>

namespace yeti {

// m rounded up to whole steps of the contractions.
__host__ __device__ constexpr int fd_m4(int m) { return (m + 3) / 4 * 4; }

// Values of a row of m that lie in the piece of vec values at k, 0 .. vec: a
// row is staged in pieces up to fd_m4(m), so that the last may lie beyond it
// altogether (two FP64 values at k = m + 1 where m is 4 j + 1).
__host__ __device__ constexpr int fd_piece(int m, int k, int vec) {
    const int left = m - k;
    return left <= 0 ? 0 : left < vec ? left : vec;
}

}  // namespace yeti
