#pragma once
#include <cuda_runtime.h>

namespace pt {

// Whether it is the faster one for these sizes.
bool gemm_skinny_better(int M, int N, int K);
// out[M, N] = x[M, K] w[N, K]^T in bf16, for few rows of x (csrc/gemm_skinny.cu). 0 or a negative error.
int gemm_skinny_nt(const void* x, const void* w, void* out, int M, int N, int K, long long lda, long long ldb, long long ldd, cudaStream_t stream);

}  // namespace pt
