// Thin SVD of small blocks by pivoted QR and one-sided Jacobi, every block of a call in one launch (svd_small.cu).
#pragma once

#include "runtime.hpp"

namespace mpsg {

struct SmallSvdBlock {
  const double* A;        // M x N, column-major
  double *U, *S, *V;      // M x k, k (descending), N x k, column-major; k = min(M, N)
  int* info;              // 1: not factorised (non-finite or extreme elements)
  int32_t M, N;
};

bool small_svd_fits(int64_t M, int64_t N);
void launch_small_svd(Context* ctx, const std::vector<SmallSvdBlock>& blocks);

}  // namespace mpsg
