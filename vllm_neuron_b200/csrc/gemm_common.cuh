// What the schedules of the weight GEMM share: operand kinds, the epilogue's operands, and the epilogue of the prompt-sized
// schedules (gemm_tcgen05.cu: decode and stream-K; gemm_pair.cu: CTA pairs).
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int GEMM_BN = 128;        // weight rows per tile  (UMMA M)
constexpr int GEMM_BK_BYTES = 128;  // one 128B swizzle row of K per stage
constexpr int KIND_WO8 = 3;         // beside UmmaKind: bf16 activations, int8 weights
template <int KIND>
struct KindTraits;
template <>
struct KindTraits<KIND_F16> {
  static constexpr int ELEM = 2, CFMT = 1, ABFMT = 1;  // bf16 in, f32 accumulate
};
template <>
struct KindTraits<KIND_F8F6F4> {
  static constexpr int ELEM = 1, CFMT = 1, ABFMT = 0;  // e4m3 in, f32 accumulate
};
template <>
struct KindTraits<KIND_I8> {
  static constexpr int ELEM = 1, CFMT = 2, ABFMT = 1;  // s8 in, s32 accumulate
};

// EPI_ROPE: EPI_LINEAR whose split-K owner epilogue also rotates q/k and scatters k/v (decode kernel, S > 1 only; gemm_small.cu); its own
// instantiation so the plain linears keep their register budget (80 vs 137)
// EPI_SILU_QUANT: EPI_SILU_MUL whose CTAs also agree on the per-token amax through a grid-wide barrier and write the
// quantised activation themselves (decode kernel, S == 1, all CTAs co-resident; fp8 of a few tokens gemm_small.cu; b200_gemm_silu_mul_quant)
enum { EPI_LINEAR = 0, EPI_SILU_MUL = 1, EPI_ROPE = 2, EPI_SILU_QUANT = 3 };

struct GemmEpilogue {
  const float* a_scale;
  const float* w_scale;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  void* out;
  int out_f32;
  float* group_amax;  // EPI_SILU_MUL: [M][N/32] max |act| over the 16 channels of each interleaved row group
  // EPI_SILU_QUANT: `out` is the quantised activation [M][N/2] (one byte per element), out_scale [M] its per-token scale;
  // fq_state = { uint64 tok_amax[128] (epoch << 32 | float bits), uint32 arrive counter, uint32 epoch }: zero once, then
  // self-maintaining (the epoch only grows, so stale maxima of earlier launches always lose the 64-bit atomicMax)
  float* out_scale;
  unsigned long long* fq_state;
  // EPI_ROPE (decode kernel with a split-K cluster only; b200_gemm_rope_kv_write): the output row is a packed qkv row
  // [Hq*D | Hkv*D | Hkv*D]; the token's owner rotates q and k (rotate-half, same roundings as rope_kv_write_kernel)
  // and scatters k, v into the block-KV pools by slot.
  struct RopeKv {
    const int64_t* positions;
    const int64_t* slot_mapping;
    const float* cos_t;
    const float* sin_t;
    __nv_bfloat16* k_pool;
    __nv_bfloat16* v_pool;
    long long num_slots;
    int max_pos, Hq, Hkv, D, bs;
  } rope;
};

// out = ((acc * a_scale) * w_scale + bias) + residual, every step rounded on its own (no FMA contraction), so that the
// decode, prefill and fused-epilogue paths produce identical bits for the same accumulator
__device__ __forceinline__ float scaled_value(float acc, float a, float w, bool has_bias, float b, bool has_res, float r) {
  float y = __fmul_rn(__fmul_rn(acc, a), w);
  if (has_bias) y = __fadd_rn(y, b);
  if (has_res) y = __fadd_rn(y, r);
  return y;
}
// SiLU(gate) * up for one channel; both inputs already rounded to bf16 like the unfused path (b200_gemm + b200_silu_mul)
__device__ __forceinline__ float silu_mul_bf16(float g, float u) {
  return __bfloat162float(__float2bfloat16_rn(silu_f32(g) * u));
}

// Prompt epilogue (stream-K; the CTA pairs have their own in gemm_pair.cuh) of one 16-token chunk, transposed through a per-warp shared-memory tile so that global
// memory sees 16-byte vectors instead of one 2-byte element per lane:
//   TMEM hands lane l the weight row n0w + l of 16 tokens; the warp writes the scaled values (a_scale, w_scale, bias
//   applied, fp32) as xp[token][row] (pitch XP_PITCH floats), then lane (token = l / 4 + 8 it, rows 8 (l % 4) ..) adds the
//   residual it loads as one 16-byte vector and stores 8 bf16 (or 8 fp32).  Per lane and chunk: 16 st.shared + 2 x
//   (2 ld.shared.v4 + ld.global.v4 + st.global.v4) instead of 16 x (4 scalar global loads + a 2-byte store) -- measured
//   on Llama-3.1-8B prefill (profiles/r02_ttft_breakdown_*.txt): o_proj 322 us, down 392 us at M = 2048 before.
// Same roundings as scaled_value().  EPI_SILU_MUL: the activation of 16 channels x 16 tokens goes through the tile as
// bf16 and leaves as one 16-byte store per lane.
constexpr int XP_PITCH = 36;                       // floats; 36 keeps the float4 reads of a quarter-warp on distinct banks
constexpr int XP_WARP_FLOATS = 16 * XP_PITCH;      // one warp's tile
template <int EPI>
__device__ __forceinline__ void epilogue_chunk_xpose(const GemmEpilogue& ep, const float (&v)[16], int m_base, int ml_base,
                                                     int M, int n0w, int N, int lane, const float* a_s, float w_sc,
                                                     float bias_v, float* xp) {
  const bool hb = ep.bias != nullptr, hr = ep.residual != nullptr;
  const int n = n0w + lane;
  const bool n_ok = n < N;
  if constexpr (EPI == EPI_LINEAR) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float y = __fmul_rn(__fmul_rn(v[j], a_s[ml_base + j]), w_sc);
      if (hb) y = __fadd_rn(y, bias_v);
      xp[j * XP_PITCH + lane] = y;
    }
    __syncwarp();
    const bool vec = (N & 7) == 0 && (reinterpret_cast<uintptr_t>(ep.out) & 15) == 0 &&
                     (!hr || (reinterpret_cast<uintptr_t>(ep.residual) & 15) == 0);
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int mm = it * 8 + (lane >> 2), c8 = (lane & 3) * 8;
      const int m = m_base + mm, nn = n0w + c8;
      if (m >= M || nn >= N) continue;
      const float4 lo = *reinterpret_cast<const float4*>(xp + mm * XP_PITCH + c8);
      const float4 hi = *reinterpret_cast<const float4*>(xp + mm * XP_PITCH + c8 + 4);
      float y[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      const int64_t off = (int64_t)m * N + nn;
      if (vec) {
        if (hr) {
          const uint4 rv = *reinterpret_cast<const uint4*>(ep.residual + off);
          const __nv_bfloat162* rh = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            y[2 * e] = __fadd_rn(y[2 * e], __low2float(rh[e]));
            y[2 * e + 1] = __fadd_rn(y[2 * e + 1], __high2float(rh[e]));
          }
        }
        if (ep.out_f32) {
          float* o = reinterpret_cast<float*>(ep.out) + off;
          *reinterpret_cast<float4*>(o) = make_float4(y[0], y[1], y[2], y[3]);
          *reinterpret_cast<float4*>(o + 4) = make_float4(y[4], y[5], y[6], y[7]);
        } else {
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(ep.out) + off) =
              make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (nn + e < N) {
            float z = y[e];
            if (hr) z = __fadd_rn(z, __bfloat162float(ep.residual[off + e]));
            if (ep.out_f32)
              reinterpret_cast<float*>(ep.out)[off + e] = z;
            else
              reinterpret_cast<__nv_bfloat16*>(ep.out)[off + e] = __float2bfloat16_rn(z);
          }
        }
      }
    }
    __syncwarp();  // the tile is rewritten by the next chunk
  } else {
    // this lane's row: gate (lane < 16) or up (lane >= 16) of channel ch; both rounded to bf16 like the unfused path
    const int I = N >> 1, n_groups = N >> 5;
    float mine[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float y = __fmul_rn(__fmul_rn(v[j], a_s[ml_base + j]), w_sc);
      if (hb) y = __fadd_rn(y, bias_v);
      mine[j] = (m_base + j < M && n_ok) ? __bfloat162float(__float2bfloat16_rn(y)) : 0.f;
    }
    const bool hi_half = lane >= 16;  // lanes < 16 finish tokens 0..7 of the chunk, lanes >= 16 finish tokens 8..15
    __nv_bfloat16* xb = reinterpret_cast<__nv_bfloat16*>(xp);  // [16 tokens][16 channels] bf16
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float send = hi_half ? mine[j] : mine[j + 8];
      const float got = __shfl_xor_sync(0xffffffffu, send, 16);
      const float g = hi_half ? got : mine[j];
      const float u = hi_half ? mine[j + 8] : got;
      const int mm = (hi_half ? 8 : 0) + j;
      const float a = silu_mul_bf16(g, u);
      xb[mm * 16 + (lane & 15)] = __float2bfloat16_rn((m_base + mm < M && n_ok) ? a : 0.f);
    }
    __syncwarp();
    {
      const int mm = lane >> 1, c8 = (lane & 1) * 8;
      const int m = m_base + mm;
      const int ch = (n0w >> 5) * 16 + c8;
      // the lane pair (2 mm, 2 mm + 1) holds the 16 channels of token mm: their maximum is the group's amax
      const uint4 val = *reinterpret_cast<const uint4*>(xb + mm * 16 + c8);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&val);
      float x = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) x = fmaxf(x, fmaxf(fabsf(__low2float(h2[e])), fabsf(__high2float(h2[e]))));
      x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
      if (m < M && n0w < N) {  // N2 % 32 == 0: a 32-row group is inside N or outside as a whole
        if ((lane & 1) == 0) ep.group_amax[(int64_t)m * n_groups + (n0w >> 5)] = x;
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(ep.out) + (int64_t)m * I + ch;
        if ((I & 7) == 0 && (reinterpret_cast<uintptr_t>(ep.out) & 15) == 0) {
          *reinterpret_cast<uint4*>(dst) = val;
        } else {
          const __nv_bfloat16* sv = reinterpret_cast<const __nv_bfloat16*>(&val);
#pragma unroll
          for (int e = 0; e < 8; ++e) dst[e] = sv[e];
        }
      }
    }
    __syncwarp();
  }
}

// Weight-only schedule of decode-sized batches (gemm_wo.cu).
// gemm_wo_wide: whether it takes a call that names no K splits.  gemm_wo_plan: its K splits and the CTAs that clusters of them hold at once.
bool gemm_wo_wide(int epi, int M, int N, int K);
int gemm_wo_plan(int epi, int M, int N, int K, int& splits, int& cap_ctas, int& stages, size_t& smem);
int launch_gemm_wo(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, cudaStream_t stream);
// Schedule on CTA pairs (gemm_pair.cu): bf16, fp8 and int8 operands.  bt: tokens of a tile; wide: how many units of two token tiles come before those
// of one.
struct PairPlan {
  int bt, wide;
};
PairPlan pair_plan(int M, int N, int K, int ab_dtype);
bool stream_k_keeps(int M, int N, int K, int ab_dtype);     // prompt-sized calls: whether stream-K takes them instead
bool pair_takes_decode(int M, int N, int K, int ab_dtype);  // up to 128 tokens: whether the pairs are faster than the decode schedule that walks all of K
void pair_shape(int M, int N, PairPlan plan, int& units, int& stages, size_t& smem);  // what the pairs walk, their ring and shared memory
int launch_gemm_pair(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, int ab_dtype, PairPlan plan,
                     cudaStream_t stream);

}  // namespace b200
