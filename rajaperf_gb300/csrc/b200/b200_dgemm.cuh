// FP64 products C = A * B on the tensor cores (dgemm_tc.cu).
#pragma once

#include "b200_internal.cuh"

namespace b200 {

// C (m x n) = A (m x k) * B (k x n), row-major.
struct Product {
  const double* A;
  const double* B;
  double* C;
  int64_t m, n, k;
};

// The tensor-core kernel takes this product (sizes only).
bool dgemm_tc_takes(const Product& p);

// One launch for one or two independent products; B200_OK or an error.
int launch_dgemm_tc(const Product* p, int count, cudaStream_t st);

}  // namespace b200
