// INT8 weight-only GEMM of decode-sized batches (M <= 128): int8 weights, bf16 activations, fp32 sums.
//
//   out[m][n] = (sum_k a[m][k] w[n][k]) * w_scale[n] + bias[n] + residual[m][n]       (or SiLU(gate) * up of interleaved rows)
//
// What bounds it is how fast TMA feeds an SM: about 3 clocks per operand row of up to 128 bytes, whatever the row holds.  A CTA of 128
// weight rows that steps 64 k at a time (gemm_tcgen05.cu) spends 128 rows on 8 KB of int8 weights and 128 more on the tokens: 0.57 us
// for 8 KB, 2.1 TB/s over the chip.  Here a CTA takes 256 weight rows and steps 128 k at a time: whole 128-byte rows of weights, and the
// token rows are shared by twice the weights, 512 rows for 32 KB.
// Two groups of eight warps take turns at widening a stage into bf16 rows in tensor memory, from where the MMAs take their A operand, one
// accumulator per 128 weight rows.  The K splits of a tile are a thread-block cluster: every CTA parks its fp32 tile in shared memory (the
// dead ring) and finishes its share of the tokens from all of them, in rank order.
// Measured (us; best of the 128-row schedule's K splits before; weight bytes at 6.65 TB/s): M = 128: 55296 x 5120 + SiLU 163 -> 97 (43),
// 5120 x 27648 108 -> 52 (21), 152064 x 5120 453 -> 245 (117), 7168 x 5120 31 -> 22 (5.5); M = 32: 55296 x 5120 139 -> 85, 152064 x 5120
// 402 -> 220.  A stage takes 1.2 us where loading alone takes 0.68; more widening warps, cheaper widening and more slots moved it by a few
// percent each.
#include <mutex>

#include "gemm_common.cuh"

namespace b200 {

constexpr int WOX_ROWS = 256;                 // weight rows of a tile
constexpr int WOX_BK = 128;                   // k of a stage
constexpr int WOX_RAW = WOX_ROWS * WOX_BK;    // bytes of raw weights per stage
constexpr int WOX_CONV = 16;                       // widening / epilogue warps: two groups of one warp per 32 rows
constexpr int WOX_THREADS = 64 + WOX_CONV * 32 + 32;  // + TMA weights, MMA, TMA activations
constexpr int WOX_MAX_ST = 5;
template <int BM>
constexpr int WOX_STAGES = BM == 128 ? 3 : BM == 64 ? 4 : WOX_MAX_ST;

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// 64 int8 -> 32 packed bf16 pairs of byte / 64, in order.  A byte + 128 in the low bits of a bf16 is the subnormal (byte + 128) 2^-133;
// times 2^127, minus 2, is byte / 64, exactly: four bytes take three instructions of the ALU pipe, which the widening fills otherwise (six
// for mask tricks: 0.34 us of a stage, ALU 64 % busy), and two of the FMA pipe.  The factor 64 goes into the channel scale.
__device__ __forceinline__ void widen_bf16(const uint4 (&raw)[4], uint32_t (&o)[32]) {
  const uint32_t k = 0x7f007f00u, c = 0xc000c000u;  // 2^127, -2
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t u = w[j] ^ 0x80808080u;
      asm("fma.rn.bf16x2 %0, %1, %2, %3;\n" : "=r"(o[i * 8 + 2 * j]) : "r"(__byte_perm(u, 0u, 0x4140)), "r"(k), "r"(c));
      asm("fma.rn.bf16x2 %0, %1, %2, %3;\n" : "=r"(o[i * 8 + 2 * j + 1]) : "r"(__byte_perm(u, 0u, 0x4342)), "r"(k), "r"(c));
    }
  }
}
constexpr float WOX_SCALE = 64.f;

template <int BM, int EPI>
__global__ void __launch_bounds__(WOX_THREADS, 1)
    gemm_wo_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map, GemmEpilogue ep, int M, int N,
                   int num_kb, int tile0) {
  constexpr int nst = WOX_STAGES<BM>;
  constexpr int A_TILE = BM * GEMM_BK_BYTES;  // 64 k of the tokens; a stage holds two
  constexpr int STAGE = WOX_RAW + 2 * A_TILE;
  constexpr uint32_t SLOT_COLS = 64;                     // 64 k of widened rows: 32 columns for each half of the tile
  constexpr uint32_t SLOTS = (512 - 2 * BM) / SLOT_COLS;  // 4 to 7, so that widening and MMAs need not take turns
  constexpr uint32_t IDESC = umma_idesc(1, 1, GEMM_BN, BM);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* part = reinterpret_cast<float*>(smem);  // [BM][256] partial sums over the dead ring
  __shared__ uint64_t full_raw[WOX_MAX_ST], empty_raw[WOX_MAX_ST], full_a[WOX_MAX_ST], empty_a[WOX_MAX_ST], full_w[SLOTS], empty_w[SLOTS], tfull;
  __shared__ uint32_t tmem_slot;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int S = (int)cluster_nctarank(), r = (int)cluster_ctarank();
  const int n_tile = tile0 + (int)blockIdx.x / S;
  const int kb0 = (int)((long long)num_kb * r / S), nk = (int)((long long)num_kb * (r + 1) / S) - kb0;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&w_map);
    tma_prefetch_desc(&a_map);
    for (int s = 0; s < nst; ++s) {
      mbar_init(&full_raw[s], 1);
      mbar_init(&empty_raw[s], WOX_CONV / 2);
      mbar_init(&full_a[s], 1);
      mbar_init(&empty_a[s], 1);
    }
    for (uint32_t t = 0; t < SLOTS; ++t) {
      mbar_init(&full_w[t], WOX_CONV / 2);
      mbar_init(&empty_w[t], 1);
    }
    mbar_init(&tfull, 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  const uint32_t tmem_base = tmem_slot, slots0 = tmem_base + 2 * BM;

  if (warp == 0) {
    // raw weights: nothing of the step writes them, so they start before the dependency resolves
    if (elect_one()) {
      const uint64_t pol = policy_evict_first();
      int s = 0, ph = 1;
      for (int i = 0; i < nk; ++i) {
        mbar_wait(&empty_raw[s], ph);
        mbar_expect_tx(&full_raw[s], WOX_RAW);
        tma_load_2d_hint(smem + (size_t)s * STAGE, &w_map, &full_raw[s], (kb0 + i) * WOX_BK, n_tile * WOX_ROWS, pol);
        if (++s == nst) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 2 + WOX_CONV) {
    if (elect_one()) {
      const uint64_t pol = policy_evict_last();
      griddep_wait();
      int s = 0, ph = 1;
      for (int i = 0; i < nk; ++i) {
        mbar_wait(&empty_a[s], ph);
        mbar_expect_tx(&full_a[s], 2 * A_TILE);
        uint8_t* dst = smem + (size_t)s * STAGE + WOX_RAW;
        tma_load_2d_hint(dst, &a_map, &full_a[s], (kb0 + i) * WOX_BK, 0, pol);
        tma_load_2d_hint(dst + A_TILE, &a_map, &full_a[s], (kb0 + i) * WOX_BK + 64, 0, pol);
        if (++s == nst) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      int s = 0, ph = 0, t = 0, pht = 0;
      for (int i = 0; i < nk; ++i) {
        mbar_wait(&full_a[s], ph);
        const uint32_t aa = smem_u32(smem + (size_t)s * STAGE + WOX_RAW);
#pragma unroll
        for (int kh = 0; kh < 2; ++kh) {
          mbar_wait(&full_w[t], pht);
          tc_fence_after();
#pragma unroll
          for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_ts_f16(tmem_base + half * BM, slots0 + t * SLOT_COLS + half * 32 + kk * 8, umma_desc_sw128(aa + kh * A_TILE + kk * 32),
                          IDESC, (uint32_t)((i | kh | kk) != 0));
          tc_commit(&empty_w[t]);
          if (kh == 1) tc_commit(&empty_a[s]);
          if (++t == (int)SLOTS) {
            t = 0;
            pht ^= 1;
          }
        }
        if (++s == nst) {
          s = 0;
          ph ^= 1;
        }
      }
      tc_commit(&tfull);
    }
    __syncwarp();
  } else {
    // widening: a thread owns one weight row of the tile, the two groups of eight warps alternate between stages.
    // A parity wait only tells a phase from the one before it.  With an odd number of stages the use of a stage before this one was the
    // other group's, and nothing this group has seen orders it behind that use's load: were that load still in flight, a wait for full_raw
    // alone would take the phase before it for its own and read stale bytes.  Hence first the wait for the MMAs of stage i - nst (empty_a):
    // they follow its widening, which followed its load.  That wait cannot come a phase late, since the MMAs of stage i need this group;
    // nor a phase early, since the MMAs, which retire in order, are past stage i - 2 nst: in stage i - 2 this group waited for those of slot
    // use 2 i - 3 - SLOTS.
    static_assert(4 * nst >= (int)SLOTS + 4, "the MMAs of stage i - 2 nst have retired when a group comes to stage i");
    const int q = warp & 3, half = ((warp - 2) >> 2) & 1, group = (warp - 2) >> 3;
    const int row = half * 128 + q * 32 + lane;
    const uint32_t lanes = (uint32_t)(q * 32) << 16;
    for (int i = group; i < nk; i += 2) {
      const int s = i % nst, use = i / nst;
      if (use) mbar_wait(&empty_a[s], (use - 1) & 1);
      mbar_wait(&full_raw[s], use & 1);
      const uint8_t* rp = smem + (size_t)s * STAGE + row * WOX_BK;
      uint4 raw[2][4];
#pragma unroll
      for (int c = 0; c < 8; ++c) raw[c >> 2][c & 3] = *reinterpret_cast<const uint4*>(rp + ((c ^ (row & 7)) << 4));  // 128B swizzle
#pragma unroll
      for (int kh = 0; kh < 2; ++kh) {
        const int h = 2 * i + kh, t = h % (int)SLOTS, turn = h / (int)SLOTS;
        uint32_t o[32];
        widen_bf16(raw[kh], o);
        if (turn) mbar_wait(&empty_w[t], (turn - 1) & 1);  // the MMAs that read this slot have retired
        __syncwarp();  // lanes may leave the wait one by one; tcgen05.st wants them together
        if (kh == 1 && lane == 0) mbar_arrive(&empty_raw[s]);  // all of the warp's rows are in registers, widened
        tc_fence_after();
        tmem_st_32x32b_x32(slots0 + lanes + t * SLOT_COLS + half * 32, o);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_w[t]);
      }
    }
    mbar_wait(&tfull, 0);
    __syncwarp();
    tc_fence_after();
#pragma unroll 1
    for (int cc = group; cc < BM / 16; cc += 2) {
      if (cc * 16 >= M) break;
      uint32_t v[16];
      tmem_ld_32x32b_x16(tmem_base + lanes + half * BM + cc * 16, v);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(cc * 16 + j) * WOX_ROWS + row] = __uint_as_float(v[j]);
    }
    griddep_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (S > 1) cluster_sync_all();  // every CTA's partial tile is in place
  if (warp >= 2 && warp < 2 + WOX_CONV) {
    const int et = threadIdx.x - 64, t4 = et & 63, tq = et >> 6;  // rows 4 t4 .. + 3, tokens tq, tq + 8, ...
    const int m_lo = M * r / S, m_hi = M * (r + 1) / S;
    const int n0 = n_tile * WOX_ROWS + 4 * t4;
    const bool hb = ep.bias != nullptr, hr = EPI == EPI_LINEAR && ep.residual != nullptr;
    const bool vec = (N & 3) == 0 && n0 + 3 < N && (!hr || (reinterpret_cast<uintptr_t>(ep.residual) & 7) == 0);
    float w4[4], b4[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      w4[e] = WOX_SCALE * (ep.w_scale && n0 + e < N ? ep.w_scale[n0 + e] : 1.f);
      b4[e] = hb && n0 + e < N ? __bfloat162float(ep.bias[n0 + e]) : 0.f;
    }
    const uint32_t mine = smem_u32(part);
#pragma unroll 2
    for (int m = m_lo + tq; m < m_hi; m += WOX_CONV / 2) {
      const uint32_t off = mine + (uint32_t)(m * WOX_ROWS + 4 * t4) * 4;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        if (p < S) {
          const float4 v = S > 1 ? ld_cluster_f4(mapa_shared(off, (uint32_t)p)) : *reinterpret_cast<const float4*>(part + m * WOX_ROWS + 4 * t4);
          sum.x += v.x;
          sum.y += v.y;
          sum.z += v.z;
          sum.w += v.w;
        }
      }
      float rs[4] = {0.f, 0.f, 0.f, 0.f};
      const int64_t o = (int64_t)m * N + n0;
      if (hr) {
        if (vec) {
          const uint2 rv = *reinterpret_cast<const uint2*>(ep.residual + o);
          const __nv_bfloat162 r01 = *reinterpret_cast<const __nv_bfloat162*>(&rv.x), r23 = *reinterpret_cast<const __nv_bfloat162*>(&rv.y);
          rs[0] = __low2float(r01), rs[1] = __high2float(r01), rs[2] = __low2float(r23), rs[3] = __high2float(r23);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (n0 + e < N) rs[e] = __bfloat162float(ep.residual[o + e]);
        }
      }
      float y[4];
      y[0] = scaled_value(sum.x, 1.f, w4[0], hb, b4[0], hr, rs[0]);
      y[1] = scaled_value(sum.y, 1.f, w4[1], hb, b4[1], hr, rs[1]);
      y[2] = scaled_value(sum.z, 1.f, w4[2], hb, b4[2], hr, rs[2]);
      y[3] = scaled_value(sum.w, 1.f, w4[3], hb, b4[3], hr, rs[3]);
      if constexpr (EPI == EPI_LINEAR) {
        if (vec && (reinterpret_cast<uintptr_t>(ep.out) & 15) == 0) {
          if (ep.out_f32)
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(ep.out) + o) = make_float4(y[0], y[1], y[2], y[3]);
          else
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(ep.out) + o) = make_uint2(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]));
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (n0 + e < N) {
              if (ep.out_f32)
                reinterpret_cast<float*>(ep.out)[o + e] = y[e];
              else
                reinterpret_cast<__nv_bfloat16*>(ep.out)[o + e] = __float2bfloat16_rn(y[e]);
            }
          }
        }
      } else {
        // 16 gate rows (lanes 8 g .. 8 g + 3), then the 16 up rows of the same channels (lanes 8 g + 4 ..); N % 32 == 0, so a group of
        // 32 rows is inside N or outside as a whole
        const int I = N >> 1, n_groups = N >> 5;
        const bool ok = n0 < N, is_gate = (lane & 4) == 0;
        float act[4], x = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float me = ok ? __bfloat162float(__float2bfloat16_rn(y[e])) : 0.f;
          const float other = __shfl_xor_sync(0xffffffffu, me, 4);
          act[e] = silu_mul_bf16(is_gate ? me : other, is_gate ? other : me);
          x = fmaxf(x, ok ? fabsf(act[e]) : 0.f);
        }
        x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
        x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
        if (ok && is_gate) {
          const int ch = (n0 >> 5) * 16 + (lane & 3) * 4;
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(ep.out) + (int64_t)m * I + ch;
          if ((reinterpret_cast<uintptr_t>(ep.out) & 7) == 0) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(act[0], act[1]), pack_bf16(act[2], act[3]));
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = __float2bfloat16_rn(act[e]);
          }
          if ((lane & 7) == 0) ep.group_amax[(int64_t)m * n_groups + (n0 >> 5)] = x;
        }
      }
    }
  }
  if (S > 1) cluster_sync_all();  // nobody leaves while a peer still reads its partial tile
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

namespace {

template <int BM>
constexpr size_t wox_smem() {
  return 1024 + (size_t)WOX_STAGES<BM> * (WOX_RAW + 2 * BM * GEMM_BK_BYTES);  // 192 to 200 KB; the partial tile takes BM KB of it
}

// K splits of `tiles` tiles: whole waves of CTAs (one per SM) of nk stages of 1.2 us each, plus filling and draining a CTA, about 4 us, and
// the exchange of the partial tiles, 2.
struct WoPlan {
  int S, cap;
  double us;
};
template <int BM, int EPI>
int plan_wo(WoPlan& best, int tiles, int num_kb) {
  static std::mutex mu;
  static int cap[9] = {};  // CTAs that clusters of S hold at once
  std::lock_guard<std::mutex> g(mu);
  auto kern = gemm_wo_kernel<BM, EPI>;
  if (!cap[1]) B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wox_smem<BM>()));
  best = {0, 0, 0.0};
  for (int S = 1; S <= 8 && S <= num_kb; ++S) {
    if (!cap[S]) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(sm_count() / S * S);
      cfg.blockDim = dim3(WOX_THREADS);
      cfg.dynamicSmemBytes = wox_smem<BM>();
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)S;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      B200_CUDA_OK(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
      cap[S] = n > 0 ? n * S : -1;
    }
    if (cap[S] < 0) continue;
    const int waves = (tiles * S + cap[S] - 1) / cap[S];
    const double us = waves * (((num_kb + S - 1) / S) * 1.2 + 4.0) + (S > 1 ? 2.0 : 0.0);
    if (!best.S || us < best.us) best = {S, cap[S], us};
  }
  B200_REQUIRE(best.S > 0, "gemm: no weight-only configuration fits");
  return B200_OK;
}

// One launch (first = 0), or `first` whole waves of uncut tiles and the rest cut along K.
template <int BM, int EPI>
int plan_launches(WoPlan& all, WoPlan& rest, int& first, int N, int K) {
  const int tiles = (N + WOX_ROWS - 1) / WOX_ROWS, num_kb = (K + WOX_BK - 1) / WOX_BK;
  int rc = plan_wo<BM, EPI>(all, tiles, num_kb);
  if (rc) return rc;
  const int main_tiles = tiles / sm_count() * sm_count();
  first = 0;
  if (main_tiles && main_tiles < tiles) {
    rc = plan_wo<BM, EPI>(rest, tiles - main_tiles, num_kb);
    if (rc) return rc;
    if (main_tiles / sm_count() * (num_kb * 1.2 + 4.0) + rest.us < all.us) first = main_tiles;
  }
  return B200_OK;
}

template <int BM, int EPI>
int launch_wo(const void* a, const void* w, const GemmEpilogue& ep, int M, int N, int K, cudaStream_t stream) {
  CUtensorMap wm, am;
  int rc = make_tmap_2d(&wm, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)K, (uint64_t)N, (uint64_t)K, WOX_BK, WOX_ROWS);
  if (rc) return rc;
  rc = make_tmap_2d(&am, a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, 64, BM);
  if (rc) return rc;
  const int tiles = (N + WOX_ROWS - 1) / WOX_ROWS, num_kb = (K + WOX_BK - 1) / WOX_BK;
  WoPlan all, rest{};
  int first;
  rc = plan_launches<BM, EPI>(all, rest, first, N, K);
  if (rc) return rc;
  auto go = [&](int tile0, int n, int S) -> int {
    B200_CUDA_OK(launch_kernel_cluster(gemm_wo_kernel<BM, EPI>, dim3(n * S), dim3(WOX_THREADS), wox_smem<BM>(), S, stream, wm, am, ep, M, N,
                                       num_kb, tile0));
    return B200_OK;
  };
  if (first) {
    rc = go(0, first, 1);
    if (rc) return rc;
  }
  return go(first, tiles - first, first ? rest.S : all.S);
}

}  // namespace

// Fewer weight rows leave most of the chip without a tile of 256, and the 128-row schedule is the faster one there.  Measured (us, 128 rows ->
// 256): linear 1024 x 1024, M = 64 6.2 -> 7.8; 2560 x 2048, M = 16 7.5 -> 7.7, 128 11.3 -> 12.3; 896 x 4864, M = 64 9.4 -> 11.7; but 2048 x 4096,
// M = 1 to 33, 0.94 to 0.99 of the time, 3072 x 2048 0.96 to 1.06, 4096 x 2048 0.97 to 1.01, 7168 x 5120 0.68; with SiLU 2048 x 4096 0.87 to
// 1.00, 1024 x 8192 0.99 to 1.07, 896 x 4864 1.05 to 1.19.
bool gemm_wo_wide(int epi, int M, int N, int K) {
  return epi == EPI_SILU_MUL ? N >= 2048 : epi == EPI_ROPE ? N >= 4096 : N >= 3072 || (N >= 2048 && K >= 4096 && M <= 32);
}

int gemm_wo_plan(int epi, int M, int N, int K, int& splits, int& cap_ctas, int& stages, size_t& smem) {
  WoPlan all{}, rest{};
  int first = 0, rc = B200_OK;
#define WO_PLAN(BM)                                                                                                                     \
  do {                                                                                                                                  \
    rc = epi == EPI_SILU_MUL ? plan_launches<BM, EPI_SILU_MUL>(all, rest, first, N, K) : plan_launches<BM, EPI_LINEAR>(all, rest, first, N, K); \
    stages = WOX_STAGES<BM>;                                                                                                            \
    smem = wox_smem<BM>();                                                                                                              \
  } while (0)
  if (M <= 32) WO_PLAN(32);
  else if (M <= 64) WO_PLAN(64);
  else WO_PLAN(128);
#undef WO_PLAN
  splits = first ? rest.S : all.S;
  cap_ctas = first ? rest.cap : all.cap;
  return rc;
}

int launch_gemm_wo(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, cudaStream_t s) {
#define WO_LAUNCH(BM) \
  return epi == EPI_SILU_MUL ? launch_wo<BM, EPI_SILU_MUL>(a, w, ep, M, N, K, s) : launch_wo<BM, EPI_LINEAR>(a, w, ep, M, N, K, s)
  if (M <= 32) WO_LAUNCH(32);
  if (M <= 64) WO_LAUNCH(64);
  WO_LAUNCH(128);
#undef WO_LAUNCH
}

}  // namespace b200
