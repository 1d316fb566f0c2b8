// The 32-bit matrix product on the tensor cores (host functions, gemm_f32_tcgen05.cu).
#pragma once

#include <cuda_runtime.h>

namespace fwb {
// Whether a matrix of N rows of K values takes it; rows 16-byte aligned, K and ldx multiples of 4.
bool gemm_f32_split_takes(int N, int K);
int gemm_f32_split(const float* X, const float* W, float* Y, const float* addend, int M, int N, int K, int ldx, int ldy,
                   cudaStream_t stream);
}  // namespace fwb
