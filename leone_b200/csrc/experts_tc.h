// The grouped products of the routed experts on tcgen05 (experts_tc.cu), called by experts.cu.
#pragma once
#include <cuda_runtime.h>

namespace leone {

constexpr int kExpertsTcMost = 256;      // experts whose tiles a block can look up

int experts_tc_product(int mode, const void* x, int ldx, const void* w, const void* w2, const int* offsets, const int* order,
                       const float* weight, int n_tokens, int experts, int top, int cols, int K, int scale_input, void* out,
                       void* sorted, int* status, cudaStream_t stream);

}  // namespace leone
