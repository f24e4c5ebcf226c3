// The schedule of the weight GEMM for a few tokens (gemm_small.cu).
#pragma once
#include "gemm_common.cuh"

namespace b200 {

// lines of 128 bytes that a warp has in flight
__host__ __device__ constexpr int small_ahead(int mma_tiles, bool wo) { return mma_tiles == 4 ? 1 : mma_tiles == 2 ? 2 : wo ? 3 : 4; }
bool gemm_small_ok(const void* a, const void* w, int epi, int M, int N, int K, int ab_dtype, int head_dim);
// What a call runs as: weight tiles of 16 rows and warps of a CTA (an SM holds 16 warps), lines that a warp has in flight.
struct SmallShape {
  int tiles, warps, lines;
};
SmallShape gemm_small_shape(int epi, int M, int N, int K, int ab_dtype);
int launch_gemm_small(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, int ab_dtype, cudaStream_t s);
// EPI_SILU_QUANT of fp8, for what gemm_small_ok takes and the chip holds at once
bool small_silu_quant_fits(int N);
int launch_gemm_small_silu_quant(const void* a, const void* w, const GemmEpilogue& ep, int M, int N, int K, cudaStream_t s);

}  // namespace b200
