// The float32 GEMM's form on the tensor cores (gemm_f32_tc.cu), as the launcher in gemm_f32.cu sees it.
#pragma once

#include <cuda_runtime.h>

namespace vx {

// Whether it takes a product: N and K decide, beside what its copies ask of the operands (rows that begin at multiples
// of 16 bytes).
bool gemm_f32_tc_takes(const float* A, const float* W, int N, int K);
// Bytes of scratch that M rows need (16-byte aligned).
long long gemm_f32_tc_scratch(int M, int K);
int gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, void* scratch, int* status,
                cudaStream_t stream);

}  // namespace vx
