// The 32-bit product on tensor cores (gemm_f32_tc.cu), called by gemm_simt.cu.
#pragma once
#include <cuda_runtime.h>

namespace leone {

// Rows of both operands start on 16 bytes.
int gemm_f32_tc(const float* a, const float* w, float* c, const float* residual, const float* bias, int m, int n, int k,
                int lda, int ldw, int ldc, int* status, cudaStream_t stream);

}  // namespace leone
