// Building blocks of the CTA-pair GEMMs (gemm_pair.cu: dense; gemm_group.cu: experts): the cta_group::2 forms of the tensor-memory,
// MMA and TMA helpers.
#pragma once
#include "gemm_common.cuh"

namespace b200 {

constexpr int PAIR_MAX_ST = 8;
constexpr int PAIR_MAX_BT = 256;

// ---- the cta_group::2 forms of the tensor-memory / MMA helpers
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(smem_slot)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
// one arrive on the barrier at this offset in BOTH CTAs once the MMAs issued so far have retired
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
// tile load into this CTA's shared memory whose bytes are counted on the LEADER's barrier (a shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tmap, uint32_t leader_bar, int32_t c0, int32_t c1,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, "
      "%4}], [%2], %5;\n" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(leader_bar), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// The same where nothing but reads of tensor memory is handed over.  Those are ordered by tcgen05.wait::ld and tcgen05.fence::before_thread_sync here and
// tcgen05.fence::after_thread_sync behind the wait, as PTX's patterns for tcgen05 between threads have it (their arrivals are relaxed too); no
// other memory goes with the arrival.  A release would first wait for the warp's stores of the chunk before.  us, released / relaxed: 4096 x 10272 x 64 in bf16
// 38.9 / 30.8, fp32 47.1 / 38.9, SiLU 50.2 / 44.1; 777 x 6144 x 4096 fp32 43.0 / 41.0, 333 x 28672 x 4096 86.0 / 84.0; long K the same.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
template <int KIND>
__device__ __forceinline__ void umma_ss_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (KIND == KIND_F16) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else if constexpr (KIND == KIND_F8F6F4) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}

// ---- epilogue of the CTA-pair schedule: tensor memory hands lane l of a warp the weight row n0w + l of 16 tokens; what the lanes hold leaves
// without passing through shared memory.  fp32 rows: a token's 32 values are a whole 128-byte line.  bf16: two tokens of a row are packed,
// neighbouring lanes swap halves, and an even lane stores two rows of the even token, an odd one of the odd token (4 bytes a lane, 64 a token);
// residuals come in the same way.  No barrier; the next chunk's accumulators and residuals are on their way while one is finished.  What bounds it is
// the latency of its dependent steps: sixteen warps instead of eight are worth as much as what was left out of them.
// A tile of 256 rows x 256 tokens takes (us, all SMs at it; eight warps and a transposing tile in shared memory / now): bf16 5.7 / 3.7, with a
// residual 15.1 / 6.5, fp32 7.1 / 4.3, SiLU 9.8 / 4.8; the main loop of a tile takes 13 at K = 2048 in bf16.
__device__ __forceinline__ uint32_t swap_halves(uint32_t own, int odd) {
  const uint32_t got = __shfl_xor_sync(0xffffffffu, own, 1);
  return __byte_perm(own, got, odd ? 0x3276 : 0x5410);
}
__device__ __forceinline__ float bf16_lo(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
// whether 16-bit rows can be stored (and read) two at a time
__device__ __forceinline__ bool epilogue_by_two(const GemmEpilogue& ep, int row) {
  return (row & 1) == 0 && ((reinterpret_cast<uintptr_t>(ep.out) | reinterpret_cast<uintptr_t>(ep.residual)) & 3) == 0;
}
// residuals of tokens m_base .. + 15: word j is of token 2 j + (lane & 1), rows n & ~1 and the next
__device__ __forceinline__ void epilogue_residual(const GemmEpilogue& ep, uint32_t (&res)[8], int m_base, int M, int n, int N, int odd) {
  const __nv_bfloat16* p = ep.residual + (int64_t)(m_base + odd) * N + (n & ~1);
#pragma unroll
  for (int j = 0; j < 8; ++j, p += 2 * (int64_t)N)
    res[j] = n < N && m_base + 2 * j + odd < M ? __ldg(reinterpret_cast<const unsigned int*>(p)) : 0u;
}
// 16 tokens; `res` as above where residuals come by two, else read here
template <int EPI>
__device__ __forceinline__ void epilogue_chunk_lanes(const GemmEpilogue& ep, const float (&v)[16], const uint32_t (&res)[8], int m_base, int M, int n0w,
                                                     int N, int lane, const float* a_s, float w_sc, float bias_v, bool scaled, bool by_two) {
  const bool hb = ep.bias != nullptr, hr = ep.residual != nullptr;
  const int n = n0w + lane, odd = lane & 1;
  float y[16];
#pragma unroll
  for (int j = 0; j < 16; j += 4) {
    const float4 a = *reinterpret_cast<const float4*>(a_s + j);
    const float as[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      y[j + e] = scaled ? __fmul_rn(__fmul_rn(v[j + e], as[e]), w_sc) : v[j + e];
      if (hb) y[j + e] = __fadd_rn(y[j + e], bias_v);
    }
  }
  if constexpr (EPI == EPI_LINEAR) {
    if (ep.out_f32 || !by_two) {
      const int left = n < N ? M - m_base : 0;
      const int64_t at = (int64_t)m_base * N + n;
      if (hr) {
        float r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = j < left ? __bfloat162float(ep.residual[at + (int64_t)j * N]) : 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) y[j] = __fadd_rn(y[j], r[j]);
      }
      if (ep.out_f32) {
        float* p = reinterpret_cast<float*>(ep.out) + at;
#pragma unroll
        for (int j = 0; j < 16; ++j, p += N)
          if (j < left) *p = y[j];
      } else {
        __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(ep.out) + at;
#pragma unroll
        for (int j = 0; j < 16; ++j, p += N)
          if (j < left) *p = __float2bfloat16_rn(y[j]);
      }
      return;
    }
    uint32_t o[8];
    if (hr) {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = swap_halves(res[j], odd);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        y[2 * j] = __fadd_rn(y[2 * j], bf16_lo(o[j]));
        y[2 * j + 1] = __fadd_rn(y[2 * j + 1], bf16_hi(o[j]));
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = swap_halves(pack_bf16(y[2 * j], y[2 * j + 1]), odd);
    __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(ep.out) + (int64_t)(m_base + odd) * N + (n & ~1);
    const int left = n < N ? M - m_base - odd : 0;
#pragma unroll
    for (int j = 0; j < 8; ++j, p += 2 * (int64_t)N)
      if (2 * j < left) *reinterpret_cast<uint32_t*>(p) = o[j];
  } else {
    // this lane's row: gate (lane < 16) or up (lane >= 16) of channel lane & 15, rounded to bf16 like the unfused path.  Lanes < 16 finish
    // tokens 0 .. 7, the others 8 .. 15.
    const int I = N >> 1, n_groups = N >> 5;
    const bool hi = lane >= 16;
    uint32_t act[4], top[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t lo8 = pack_bf16(y[2 * j], y[2 * j + 1]), hi8 = pack_bf16(y[2 * j + 8], y[2 * j + 9]);
      const uint32_t got = __shfl_xor_sync(0xffffffffu, hi ? lo8 : hi8, 16);
      const uint32_t g = hi ? got : lo8, u = hi ? hi8 : got;
      act[j] = pack_bf16(silu_mul_bf16(bf16_lo(g), bf16_lo(u)), silu_mul_bf16(bf16_hi(g), bf16_hi(u)));
      top[j] = act[j] & 0x7fff7fffu;
    }
    const int t0 = m_base + (hi ? 8 : 0);
    const bool n_ok = n0w < N;  // N % 32 == 0: a 32-row group is inside N or outside as a whole
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(ep.out) + (n0w >> 5) * 16;
    if (by_two) {
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = swap_halves(act[j], odd);
      __nv_bfloat16* p = out + (int64_t)(t0 + odd) * I + (lane & 14);
#pragma unroll
      for (int j = 0; j < 4; ++j, p += 2 * (int64_t)I)
        if (n_ok && t0 + 2 * j + odd < M) *reinterpret_cast<uint32_t*>(p) = o[j];
    } else if (n_ok) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (t0 + j < M) out[(int64_t)(t0 + j) * I + (lane & 15)] = __float2bfloat16_rn(j & 1 ? bf16_hi(act[j >> 1]) : bf16_lo(act[j >> 1]));
    }
    // the 16 channels' maxima of each token: halving over the lanes, two tokens a word
    auto max2 = [](uint32_t a, uint32_t b) {
      const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
      return *reinterpret_cast<const uint32_t*>(&m);
    };
    const bool b8 = lane & 8, b4 = lane & 4;
    uint32_t m0 = max2(b8 ? top[2] : top[0], __shfl_xor_sync(0xffffffffu, b8 ? top[0] : top[2], 8));
    uint32_t m1 = max2(b8 ? top[3] : top[1], __shfl_xor_sync(0xffffffffu, b8 ? top[1] : top[3], 8));
    m0 = max2(b4 ? m1 : m0, __shfl_xor_sync(0xffffffffu, b4 ? m0 : m1, 4));
    m0 = max2(m0, __shfl_xor_sync(0xffffffffu, m0, 2));
    m0 = max2(m0, __shfl_xor_sync(0xffffffffu, m0, 1));
    const int t = t0 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + odd;
    if ((lane & 2) == 0 && n_ok && t < M) ep.group_amax[(int64_t)t * n_groups + (n0w >> 5)] = odd ? bf16_hi(m0) : bf16_lo(m0);
  }
}

// the loads of v have arrived (and nothing reads it before)
__device__ __forceinline__ void tmem_ld_wait16(uint32_t (&a)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]), "+r"(a[8]), "+r"(a[9]), "+r"(a[10]),
                 "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])::"memory");
}

}  // namespace b200
