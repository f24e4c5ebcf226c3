// What the sequential state-space scan (ssm_scan.cu) and its segments as matrix products (ssm_segment.cu) share.
#pragma once
#include "hybrid_common.cuh"

namespace b200 {

enum { SEG_FIRST = 1, SEG_LAST = 2 };
constexpr int SEG_TOKENS = 128;  // most tokens of a segment that the matrix form takes
// a sequence that is one segment of a few tokens (decoded ones beside prompt portions): the sequential kernel reads and writes its state
// once, where the matrix form would take it through scratch
constexpr int SEG_SHORT = 32;
__device__ __forceinline__ bool seg_is_short(int4 sd) { return (sd.w & (SEG_FIRST | SEG_LAST)) == (SEG_FIRST | SEG_LAST) && sd.y - sd.x <= SEG_SHORT; }

// whether the matrix form takes these operands
bool ssd_segments_ok(const void* xbc, int x_dtype, int C, const float* state, int P, int N, const float* seg_state, const float* y);
// every segment's own state (from zero) and summed step size -> scratch; then, once the scratch holds the start states
// (ssd_seg_combine_kernel), outputs and the slots' new states
int ssd_segment_states(const void* xbc, int C, const float* dt_in, int ld_dt, int dt_col0, const float* A_log, const float* dt_bias, int H,
                       int P, int N, int G, const int32_t* segs, int num_segs, const int32_t* seq_seg0, float* seg_state, float* seg_dtsum,
                       cudaStream_t st);
int ssd_segment_outputs(const void* xbc, int C, const float* dt_in, int ld_dt, int dt_col0, const float* A_log, const float* dt_bias,
                        const float* D, float* state, const int32_t* seq_slot, const int32_t* seq_pos0, float* y, int B, int H, int P, int N,
                        int G, const int32_t* segs, int num_segs, const int32_t* seq_seg0, const float* seg_state, const float* seg_dtsum,
                        cudaStream_t st);

}  // namespace b200
