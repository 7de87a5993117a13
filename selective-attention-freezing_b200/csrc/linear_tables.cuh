// The row selection of an indexed linear as the CUDA-core and split fp32 kernels read it: weights in place, selected rows
// n = g * slab + r at row (row0[g] + r) of matrix weight[g].
#pragma once
#include <string.h>

#include "saf_internal.h"

namespace saf {

constexpr int MAX_SLABS = 2048;
struct SlabTable {
  int32_t row0[MAX_SLABS];
  uint8_t weight[MAX_SLABS];
  uint8_t rope[MAX_SLABS];
};
struct WeightSet {
  const void* w[SAF_MAX_WEIGHTS];
  const void* b[SAF_MAX_WEIGHTS];
  int64_t ldw[SAF_MAX_WEIGHTS];
  int64_t cdw[SAF_MAX_WEIGHTS];
};

// pointer to element (row n of the selection, column c)
template <typename T>
__device__ __forceinline__ const T* welem(const WeightSet& ws, const SlabTable& tb, int n, int slab, int c) {
  const int g = n / slab, r = n - g * slab;
  const int w = tb.weight[g];
  return reinterpret_cast<const T*>(ws.w[w]) + (int64_t)(tb.row0[g] + r) * ws.ldw[w] + (int64_t)c * ws.cdw[w];
}

// fp32 products on rows of whole 16-byte pieces (linear_f32_sm100.cu).  mode 0: out = x W^T, A = x; 1: dx = dout W,
// A = dout, X = bias over the columns or null; 2: dW = dout^T x, A = dout, X = x, results through the weight addresses
int launch_linear_f32(int mode, const void* A, int64_t lda, const void* X, int64_t ldx, void* Cout, int64_t ldc,
                      const SafIndexedLinearArgs& a, const WeightSet& ws, const SlabTable& tb, cudaStream_t st);

}  // namespace saf
