// What the experts' sort (moe.cu) hands to the products over sorted rows (gemm_pair_tcgen05.cu).
#pragma once

#include <cuda_runtime.h>

namespace ifx {

constexpr int kItemTokens = 256;         // token rows of a tile at most

// One tile of token rows: the matrix of the stack that it takes, its first row, how many rows are its own, and that number
// rounded up to a multiple of 32.  Entry 0 of a list holds the number of tiles in `matrix`.
struct __align__(16) PairItem {
  int matrix, row, count, width;
};

}  // namespace ifx
