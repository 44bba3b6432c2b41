// True fp32 products: fk_gemm_f32 and the fp32 form of fk_group_gemm.
#pragma once

#include "fk_common.cuh"

namespace fk {

struct F32Product {
  const float* x; int64_t x_stride, x_group;
  const float* w; int64_t w_rows;              // weight rows per group (n, or 2 n)
  const float* bias;                           // [w_rows] or null
  float* y; int64_t y_stride, y_group;
  const int32_t* offsets; const int32_t* gather;   // row groups (null: column groups)
  int64_t rows, x_rows;
  int groups, n, k, act;                       // act < 0: plain products
  int32_t* status;
};

// Rows of x and w are 16-byte aligned, k a multiple of 4, sizes within 31 bits and at most 65535
// groups.
int launch_f32_product(const F32Product& p, cudaStream_t stream);

}  // namespace fk
