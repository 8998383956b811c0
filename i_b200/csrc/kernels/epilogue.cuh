// The caller's pointwise operators on one value of a result that is not produced in tiles (folds,
// dot products): the arithmetic of the pointwise kernels, one operator after the other.
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace ib {

static __device__ __noinline__ float epilogue_value(const GemmEpilogue& e, float v, size_t row, size_t col, size_t cols) {
#pragma unroll 1
  for (int k = 0; k < e.n_ops; ++k) {
    const int w = e.which[k];
    if (w < 0) {
      v = apply_unary(e.op[k], v);
      continue;
    }
    const float* p = e.operand[w];
    const int mode = e.mode[w];
    const float t = __ldg(mode == 0 ? p + row * cols + col : mode == 1 ? p + row : mode == 2 ? p + col : p);
    v = e.acc_right[k] ? apply_binary(e.op[k], t, v) : apply_binary(e.op[k], v, t);
  }
  return v;
}

}  // namespace ib
