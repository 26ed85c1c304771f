// The product kernel for few columns (skinny.cu), as spmm.cu launches it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vb {

struct SkinnyParams {
  const uint8_t* tiles;
  const int32_t* tile_cols;
  const int32_t* row_ptr;
  const float* row_scale;   // or null
  const uint8_t* b;         // [K, N], or [N, K] when transposed
  long long ldb;            // bytes
  int K, N, M;
  const float* col_scale;
  float b_scale;
  const float* bias;
  const float* row_bias;
  void* out;
  long long ldc;
  int out_dtype, act, terms, a_stable;
};

cudaError_t skinny_launch(const SkinnyParams& p, int kind, bool transposed, int nbr, long long nnz, cudaStream_t st);

}  // namespace vb
