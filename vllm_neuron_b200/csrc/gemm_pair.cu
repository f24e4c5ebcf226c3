// Weight GEMM of prompt-sized batches (M > 128) on CTA pairs:
//
//   out[m][n] = (sum_k a[m][k] w[n][k]) * a_scale[m] * w_scale[n] + bias[n] + residual[m][n]
//
// A cluster of two CTAs computes a tile of 256 weight rows x `bt` tokens with tcgen05.mma.cta_group::2: each CTA stages its own
// 128 weight rows and half of the tokens, the leader's elected thread issues the MMAs for both, and each CTA's tensor memory ends up
// with its 128 weight rows x all bt tokens.  Each operand row crosses the L2 -> SM path once per pair tile, 512 rows for 256 x 256 x 64
// multiply-adds, where a single-CTA tile of 128 x 256 takes 384 for half as many; and that path is what bounds this kernel: 32 KB
// per CTA and k-block in 0.39 us, 84 GB/s per SM, 12.4 TB/s over the chip, whatever the ring depth from 4 stages on (2 stages are
// slower, and boxes of half the rows, from one or four issuing warps, take 0.53 us).  Pairs are persistent over whole tiles, K is
// not cut: two accumulators of 256 columns alternate, so a tile's epilogue runs under the next tile's MMAs.
// Measured against the stream-K schedule that it replaces for these operand kinds (us, B200): bf16 4096 x 10272 x 2048 183 -> 135,
// 4096 x 2048 x 2048 73 -> 32, 777 x 28672 x 4096 + SiLU 248 -> 175, 333 x 2048 x 2048 71 -> 15; fp8 2048 x 28672 x 4096 + SiLU
// 316 -> 195, 2048 x 4096 x 14336 145 -> 94 (2.5 PFLOP/s).
// fp32 outputs against 64 bits (2-norm, bf16 normal operands): the tensor cores cut the low bits of every sum of 16 products, so the error
// grows with the length of a sum that is not cut: K = 4096 4.4e-6 (stream-K 3.7e-6 at 2048 x 4096, where it cuts few tiles, 1.6e-6 at 777 x
// 2048), K = 14336 1.6e-5 (1.4e-5, 6.0e-6); a quarter to one percent of a bf16 output's own rounding, 1.7e-3.  Spans of four k-blocks added in
// registers bring 2.4e-7 at any K, take 15 to 60 % longer, and leave the error of every serving step as it is.
#include <mutex>

#include "gemm_pair.cuh"

namespace b200 {

// Warp roles: 0 = TMA producer (both CTAs), 1 = tensor-memory owner (both) and MMA issuer (leader), 2..9 = epilogue.
template <int KIND, int EPI>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map, GemmEpilogue ep, int M, int N,
                     int m_tiles, int tiles, int num_kb, int bt, int nst, int w_stream_once) {
  using T = KindTraits<KIND>;
  constexpr int BK_ELEMS = GEMM_BK_BYTES / T::ELEM;
  constexpr int W_TILE = GEMM_BN * GEMM_BK_BYTES;
  const int a_tile = (bt >> 1) * GEMM_BK_BYTES;  // this CTA's half of the tokens
  const int stage = W_TILE + a_tile;
  const uint32_t idesc = umma_idesc(T::CFMT, T::ABFMT, 2 * GEMM_BN, (uint32_t)bt);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[PAIR_MAX_ST], empty[PAIR_MAX_ST], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float a_s_tile[PAIR_MAX_BT];
  __shared__ __align__(16) float xpose[PAIR_EPI_WARPS * XP_WARP_FLOATS];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&w_map);
    tma_prefetch_desc(&a_map);
    for (int s = 0; s < nst; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 2 * PAIR_EPI_WARPS);
    }
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_slot, 2 * PAIR_MAX_BT);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before either signals the other's
  tc_fence_after();
  griddep_launch();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t pol_w = w_stream_once ? policy_evict_first() : policy_evict_last();
      const uint64_t pol_a = policy_evict_last();  // activations are re-read by every pair
      const int n_off = (int)rank * GEMM_BN, m_off = (int)rank * (bt >> 1);
      // weights do not depend on any kernel of the step: fill the ring with the first tile's before the dependency resolves
      const int npre = num_kb < nst ? num_kb : nst;
      for (int i = 0; i < npre; ++i) {
        if (rank == 0) mbar_expect_tx(&full[i], 2 * stage);
        tma_load_2d_pair(smem + (size_t)i * stage, &w_map, mapa_shared(smem_u32(&full[i]), 0), i * BK_ELEMS,
                         (pair / m_tiles) * 2 * GEMM_BN + n_off, pol_w);
      }
      griddep_wait();
      int i = 0, s = 0, ph = 1;  // first pass over the ring: the stages are free (a parity-1 wait on a fresh barrier returns at once)
      for (int tile = pair; tile < tiles; tile += pairs) {
        const int n0 = (tile / m_tiles) * 2 * GEMM_BN + n_off, m0 = (tile % m_tiles) * bt + m_off;
        for (int kb = 0; kb < num_kb; ++kb, ++i) {
          const uint32_t bar = mapa_shared(smem_u32(&full[s]), 0);
          uint8_t* ws = smem + (size_t)s * stage;
          if (i >= npre) {
            mbar_wait(&empty[s], ph);
            if (rank == 0) mbar_expect_tx(&full[s], 2 * stage);
            tma_load_2d_pair(ws, &w_map, bar, kb * BK_ELEMS, n0, pol_w);
          }
          tma_load_2d_pair(ws + W_TILE, &a_map, bar, kb * BK_ELEMS, m0, pol_a);
          if (++s == nst) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      int s = 0, ph = 0, seg = 0;
      for (int tile = pair; tile < tiles; tile += pairs, ++seg) {
        const int as = seg & 1;
        if (seg >= 2) mbar_wait(&tempty[as], ((seg >> 1) - 1) & 1);
        tc_fence_after();
        const uint32_t acc = tmem_base + (uint32_t)(as * PAIR_MAX_BT);
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(&full[s], ph);
          tc_fence_after();
          if (lane == 0) {
            const uint32_t wa = smem_u32(smem + (size_t)s * stage), aa = wa + W_TILE;
#pragma unroll
            for (int kk = 0; kk < GEMM_BK_BYTES / 32; ++kk)  // UMMA_K = 32 bytes of K
              umma_ss_pair<KIND>(acc, umma_desc_sw128(wa + kk * 32), umma_desc_sw128(aa + kk * 32), idesc, (uint32_t)((kb | kk) != 0));
            tc_commit_pair(&empty[s]);
          }
          __syncwarp();
          if (++s == nst) {
            s = 0;
            ph ^= 1;
          }
        }
        if (lane == 0) tc_commit_pair(&tfull[as]);
        __syncwarp();
      }
    }
  } else {
    const int lg = warp & 3, half = (warp - 2) >> 2;
    const int et = threadIdx.x - 64;
    float* xp = xpose + (warp - 2) * XP_WARP_FLOATS;
    griddep_wait();
    int seg = 0;
    for (int tile = pair; tile < tiles; tile += pairs, ++seg) {
      const int as = seg & 1;
      const int m0 = (tile % m_tiles) * bt;
      const int n0w = (tile / m_tiles) * 2 * GEMM_BN + (int)rank * GEMM_BN + lg * 32;
      const int n = n0w + lane;
      named_bar_sync(1, 32 * PAIR_EPI_WARPS);  // the previous tile's readers of a_s_tile are done
      if (et < bt) a_s_tile[et] = (ep.a_scale && m0 + et < M) ? ep.a_scale[m0 + et] : 1.f;
      const float w_sc = (ep.w_scale && n < N) ? ep.w_scale[n] : 1.f;
      const float bias_v = (ep.bias && n < N) ? __bfloat162float(ep.bias[n]) : 0.f;
      named_bar_sync(1, 32 * PAIR_EPI_WARPS);
      mbar_wait(&tfull[as], (seg >> 1) & 1);
      __syncwarp();  // lanes may leave the wait one by one; tcgen05.ld wants them together
      tc_fence_after();
      const uint32_t acc = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(as * PAIR_MAX_BT);
      // the two warps of a lane group take alternate pairs of 16-token chunks
#pragma unroll 1
      for (int c0 = half * 32; c0 < bt; c0 += 64) {
        uint32_t v0[16], v1[16];
        tmem_ld_32x32b_x16(acc + c0, v0);
        tmem_ld_32x32b_x16(acc + c0 + 16, v1);
        tmem_ld_wait();
        float f[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) f[j] = KIND == KIND_I8 ? (float)(int32_t)v0[j] : __uint_as_float(v0[j]);
        if (m0 + c0 < M) epilogue_chunk_xpose<EPI>(ep, f, m0 + c0, c0, M, n0w, N, lane, a_s_tile, w_sc, bias_v, xp);
#pragma unroll
        for (int j = 0; j < 16; ++j) f[j] = KIND == KIND_I8 ? (float)(int32_t)v1[j] : __uint_as_float(v1[j]);
        if (m0 + c0 + 16 < M) epilogue_chunk_xpose<EPI>(ep, f, m0 + c0 + 16, c0 + 16, M, n0w, N, lane, a_s_tile, w_sc, bias_v, xp);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[as]), 0));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // nobody leaves, or frees tensor memory, while the other CTA's MMAs or arrivals may still reach it
  if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * PAIR_MAX_BT);
}

namespace {

constexpr size_t PAIR_SMEM_RING = 232448 - 1024 - (PAIR_MAX_BT * 4 + PAIR_EPI_WARPS * XP_WARP_FLOATS * 4 + 512);

int pair_stages(int bt) {
  int n = (int)(PAIR_SMEM_RING / (size_t)(GEMM_BN * GEMM_BK_BYTES + (bt / 2) * GEMM_BK_BYTES));
  return n > PAIR_MAX_ST ? PAIR_MAX_ST : n;
}

// how many CTA pairs the chip holds at once (one CTA per SM; an odd SM of a cluster domain stays empty)
template <int KIND, int EPI>
int max_pairs(int& out) {
  static std::mutex mu;
  static int pairs = 0;
  std::lock_guard<std::mutex> g(mu);
  if (!pairs) {
    auto kern = gemm_pair_kernel<KIND, EPI>;
    B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(PAIR_SMEM_RING + 1024)));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(sm_count());
    cfg.blockDim = dim3(PAIR_THREADS);
    cfg.dynamicSmemBytes = PAIR_SMEM_RING + 1024;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    B200_CUDA_OK(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    B200_REQUIRE(n > 0, "gemm: no CTA pair fits this device");
    pairs = n;
  }
  out = pairs;
  return B200_OK;
}

template <int KIND, int EPI>
int launch_pair(const void* a, const void* w, const GemmEpilogue& ep, int M, int N, int K, int bt, cudaStream_t stream) {
  constexpr int EB = KindTraits<KIND>::ELEM, BK = GEMM_BK_BYTES / EB;
  const CUtensorMapDataType dt = EB == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  int pairs = 0;
  int rc = max_pairs<KIND, EPI>(pairs);
  if (rc) return rc;
  CUtensorMap wm, am;
  rc = make_tmap_2d(&wm, w, dt, EB, (uint64_t)K, (uint64_t)N, (uint64_t)K * EB, BK, GEMM_BN);
  if (rc) return rc;
  rc = make_tmap_2d(&am, a, dt, EB, (uint64_t)K, (uint64_t)M, (uint64_t)K * EB, BK, bt / 2);
  if (rc) return rc;
  const int m_tiles = (M + bt - 1) / bt, n_tiles = (N + 2 * GEMM_BN - 1) / (2 * GEMM_BN), tiles = m_tiles * n_tiles;
  const int used = tiles < pairs ? tiles : pairs;
  B200_CUDA_OK(launch_kernel_cluster(gemm_pair_kernel<KIND, EPI>, dim3(2 * used), dim3(PAIR_THREADS), PAIR_SMEM_RING + 1024, 2, stream, wm,
                                     am, ep, M, N, m_tiles, tiles, (K + BK - 1) / BK, bt, pair_stages(bt), m_tiles == 1 ? 1 : 0));
  return B200_OK;
}

}  // namespace

// Tokens of a tile.  A wave of tiles costs its k-blocks -- 640 clocks up to 128 tokens, from there 3 for each of the 128 + bt/2 operand
// rows (measured: 0.336 us at 96 and 128 tokens, 0.358 at 192, 0.428 at 256) -- plus filling the ring, draining the last accumulator and
// the launch; so the widest tile wins unless a narrower one saves a wave or the padding of the last token tile.  Measured (us, 74 pairs):
//   4096 x 10272 x 2048 bf16: bt 256 134.8, 224 149.2, 192 160.7, 128 212.6;  3688 x 2048 x 2048: 256 31.2, 192 41.8;
//   1636 x 2048 x 2048: 192 18.6, 256 19.3, 128 28.5;  333 x 2048 x 2048: 64 15.2, 256 17.8;  777 x 4096 x 4096: 224 29.9, 192 50.8.
// 0: stream-K (gemm_tcgen05.cu) takes the call.  It cuts K, which pays where few tiles walk a long K or a nearly empty wave follows a full
// one: about 25 us, 0.52 for each k-block of 128 x 256 of an SM's share, and 8 for every CTA that adds to one tile.  Measured (us, pairs /
// stream-K, bf16): 129 x 5120 x 27648 152 / 106, 256 158 / 115, 320 158 / 156, 512 164 / 173, 777 327 / 292, 1290 400 / 447;
// 300 x 1024 x 28672 155 / 123, 1400 157 / 122; 200 x 8192 x 28672 175 / 139, 300 170 / 240; 129 x 4096 x 14336 80 / 85, 1200 161 / 158.
// Over 700 measured calls (bf16 and fp8, 129 to 4096 tokens) the rule takes the slower side by more than 5 % in seven, by 13 % at most, and
// never leaves a faster pair schedule.
int pair_tokens(int M, int N, int K, int ab_dtype) {
  const int eb = ab_dtype == B200_BF16 ? 2 : 1, sms = sm_count();
  const int pairs = sms / 2, num_kb = (K * eb + GEMM_BK_BYTES - 1) / GEMM_BK_BYTES, n_tiles = (N + 2 * GEMM_BN - 1) / (2 * GEMM_BN);
  long long best_cost = 0;
  int best = 0;
  for (int bt = PAIR_MAX_BT; bt >= 64; bt -= 32) {
    const long long tiles = (long long)((M + bt - 1) / bt) * n_tiles, waves = (tiles + pairs - 1) / pairs;
    const long long cost = waves * ((long long)num_kb * (bt <= 128 ? 640 : 3 * (GEMM_BN + bt / 2)) + 2500 + 10 * bt);
    if (!best || cost < best_cost) {
      best = bt;
      best_cost = cost;
    }
  }
  const double sk_tiles = (double)((M + 255) / 256) * ((N + GEMM_BN - 1) / GEMM_BN), shared = sms / sk_tiles;
  const double stream_k_us = 25.0 + 0.52 * sk_tiles * num_kb / sms + 8.0 * (shared > 1.0 ? shared : 1.0);
  return stream_k_us * 1850.0 < (double)best_cost ? 0 : best;  // clocks at 1.85 GHz
}

int launch_gemm_pair(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, int ab_dtype, int bt,
                     cudaStream_t s) {
  if (ab_dtype == B200_BF16)
    return epi == EPI_SILU_MUL ? launch_pair<KIND_F16, EPI_SILU_MUL>(a, w, ep, M, N, K, bt, s)
                               : launch_pair<KIND_F16, EPI_LINEAR>(a, w, ep, M, N, K, bt, s);
  if (ab_dtype == B200_FP8_E4M3)
    return epi == EPI_SILU_MUL ? launch_pair<KIND_F8F6F4, EPI_SILU_MUL>(a, w, ep, M, N, K, bt, s)
                               : launch_pair<KIND_F8F6F4, EPI_LINEAR>(a, w, ep, M, N, K, bt, s);
  return epi == EPI_SILU_MUL ? launch_pair<KIND_I8, EPI_SILU_MUL>(a, w, ep, M, N, K, bt, s)
                             : launch_pair<KIND_I8, EPI_LINEAR>(a, w, ep, M, N, K, bt, s);
}

}  // namespace b200
