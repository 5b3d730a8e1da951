// Float32 matrix product on the tensor cores (gemm_f32_tc.cu).
#pragma once
#include <cuda_runtime.h>

// out[M, N] = a[M, K] . w[N, K]^T, all float32 and dense, K > 0; a wait that expires sets a bit of `err`.
int xb_gemm_f32_tc(float* out, const float* a, const float* w, int M, int N, int K, int* err, cudaStream_t stream);
