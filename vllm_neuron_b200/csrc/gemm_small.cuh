// The schedule of the weight GEMM for a few tokens (gemm_small.cu).
#pragma once
#include "gemm_common.cuh"

namespace b200 {

bool gemm_small_ok(const void* a, const void* w, int epi, int M, int N, int K, int ab_dtype, int head_dim);
int launch_gemm_small(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, int ab_dtype, cudaStream_t s);

}  // namespace b200
