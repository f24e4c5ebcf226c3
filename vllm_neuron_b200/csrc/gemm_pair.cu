// Weight GEMM on CTA pairs: prompt-sized batches (M > 128) but those that stream_k_keeps, and decode-sized ones that pair_takes_decode:
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
// Since operand rows are what bounds it, a pair may also take two neighbouring token tiles of one weight tile at once, both accumulators
// full: 384 rows for 512 tokens instead of twice 256 (figures at pair_plan); the next unit's first token tile runs ahead through the ring (and the
// ring fills on) while the epilogue drains the other accumulator.  The sums are the same, bit for bit: K goes into one accumulator in one order.
// Measured against the stream-K schedule that it replaces for these operand kinds (us, B200): bf16 4096 x 10272 x 2048 183 -> 135,
// 4096 x 2048 x 2048 73 -> 32, 777 x 28672 x 4096 + SiLU 248 -> 175, 333 x 2048 x 2048 71 -> 15; fp8 2048 x 28672 x 4096 + SiLU
// 316 -> 195, 2048 x 4096 x 14336 145 -> 94 (2.5 PFLOP/s).
// fp32 outputs against 64 bits (2-norm, bf16 normal operands): the tensor cores cut the low bits of every sum of 16 products, so the error
// grows with the length of a sum that is not cut: K = 4096 4.4e-6 (stream-K 3.7e-6 at 2048 x 4096, where it cuts few tiles, 1.6e-6 at 777 x
// 2048), K = 14336 1.6e-5 (1.4e-5, 6.0e-6); a quarter to one percent of a bf16 output's own rounding, 1.7e-3.  Spans of four k-blocks added in
// registers bring 2.4e-7 at any K, take 15 to 60 % longer, and leave the error of every serving step as it is.
#include <limits.h>

#include <mutex>

#include "gemm_pair.cuh"

namespace b200 {

constexpr int PAIR_EPI_WARPS = 16;                     // four per 32-lane group of tensor memory: they share its token chunks
constexpr int PAIR_THREADS = 64 + 32 * PAIR_EPI_WARPS;  // + the TMA producer and the MMA issuer

// What a pair walks: `wide` units of two neighbouring token tiles of one weight tile, which share its weight rows (both accumulators at
// once), then the token tiles that are left one by one.
struct PairUnits {
  int mt, wide, lone0, units;  // token tiles; wide units; token tiles (weight tile by weight tile) that they cover; all units
  __host__ __device__ PairUnits(int mt_, int n_tiles, int wide_) : mt(mt_), wide(wide_) {
    const int u = (mt + 1) / 2, r = wide % u;  // a weight tile's last wide unit holds one token tile where their number is odd
    lone0 = wide / u * mt + (2 * r < mt ? 2 * r : mt);
    units = wide + n_tiles * mt - lone0;
  }
  // -> weight tile, first token tile, number of token tiles
  __device__ __forceinline__ void at(int i, int& nt, int& m, int& cnt) const {
    if (i < wide) {
      const int u = (mt + 1) / 2;
      nt = i / u;
      m = 2 * (i - nt * u);
      cnt = mt - m < 2 ? 1 : 2;
    } else {
      const int t = lone0 + i - wide;
      nt = t / mt;
      m = t - nt * mt;
      cnt = 1;
    }
  }
};

// Warp roles: 0 = TMA producer (both CTAs), 1 = tensor-memory owner (both) and MMA issuer (leader), 2..17 = epilogue.
template <int KIND, int EPI>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map, GemmEpilogue ep, int M, int N,
                     PairUnits un, int num_kb, int bt, int nst, int stage, int w_stream_once) {
  using T = KindTraits<KIND>;
  constexpr int BK_ELEMS = GEMM_BK_BYTES / T::ELEM;
  constexpr int W_TILE = GEMM_BN * GEMM_BK_BYTES;
  const int a_tile = (bt >> 1) * GEMM_BK_BYTES;  // this CTA's half of a token tile
  const uint32_t idesc = umma_idesc(T::CFMT, T::ABFMT, 2 * GEMM_BN, (uint32_t)bt);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[PAIR_MAX_ST], empty[PAIR_MAX_ST], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float a_s_tile[PAIR_MAX_BT];

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
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
    if (elect_one()) {
      const uint64_t pol_w = w_stream_once ? policy_evict_first() : policy_evict_last();
      const uint64_t pol_a = policy_evict_last();  // activations are re-read by every pair
      const int n_off = (int)rank * GEMM_BN, m_off = (int)rank * (bt >> 1);
      int nt, mt, cnt;
      un.at(pair, nt, mt, cnt);
      // weights do not depend on any kernel of the step: fill the ring with the first unit's before the dependency resolves
      const int npre = num_kb < nst ? num_kb : nst;
      for (int i = 0; i < npre; ++i) {
        if (rank == 0) mbar_expect_tx(&full[i], 2 * (W_TILE + cnt * a_tile));
        tma_load_2d_pair(smem + (size_t)i * stage, &w_map, mapa_shared(smem_u32(&full[i]), 0), i * BK_ELEMS, nt * 2 * GEMM_BN + n_off, pol_w);
      }
      griddep_wait();
      int i = 0, s = 0, ph = 1;  // first pass over the ring: the stages are free (a parity-1 wait on a fresh barrier returns at once)
      for (int unit = pair; unit < un.units; unit += pairs) {
        un.at(unit, nt, mt, cnt);
        const int n0 = nt * 2 * GEMM_BN + n_off, m0 = mt * bt + m_off;
        for (int kb = 0; kb < num_kb; ++kb, ++i) {
          const uint32_t bar = mapa_shared(smem_u32(&full[s]), 0);
          uint8_t* ws = smem + (size_t)s * stage;
          if (i >= npre) {
            mbar_wait(&empty[s], ph);
            if (rank == 0) mbar_expect_tx(&full[s], 2 * (W_TILE + cnt * a_tile));
            tma_load_2d_pair(ws, &w_map, bar, kb * BK_ELEMS, n0, pol_w);
          }
          tma_load_2d_pair(ws + W_TILE, &a_map, bar, kb * BK_ELEMS, m0, pol_a);
          if (cnt == 2) tma_load_2d_pair(ws + W_TILE + a_tile, &a_map, bar, kb * BK_ELEMS, m0 + bt, pol_a);
          if (++s == nst) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int s = 0, ph = 0, seg = 0, nt, mt, cnt;
      // the MMAs of token tile h of the unit whose operands lie in stage `st`
      auto mma = [&](int st, int h, uint32_t acc, bool first) {
        const uint32_t wa = smem_u32(smem + (size_t)st * stage), aa = wa + W_TILE + h * a_tile;
#pragma unroll
        for (int kk = 0; kk < GEMM_BK_BYTES / 32; ++kk)  // UMMA_K = 32 bytes of K
          umma_ss_pair<KIND>(acc, umma_desc_sw128(wa + kk * 32), umma_desc_sw128(aa + kk * 32), idesc, (uint32_t)(!first || kk != 0));
      };
      for (int unit = pair; unit < un.units; unit += pairs) {
        un.at(unit, nt, mt, cnt);
        const int as = seg & 1;
        if (seg >= 2) mbar_wait(&tempty[as], ((seg >> 1) - 1) & 1);
        tc_fence_after();
        const uint32_t acc = tmem_base + (uint32_t)(as * PAIR_MAX_BT), acc2 = tmem_base + (uint32_t)((as ^ 1) * PAIR_MAX_BT);
        // of a wide unit the first token tile runs ahead through the ring while the epilogue still drains the other accumulator
        int ahead = 0, s2 = s;
        if (cnt == 2) {
          for (; ahead < num_kb && ahead < nst; ++ahead) {
            mbar_wait(&full[s], ph);
            tc_fence_after();
            mma(s, 0, acc, ahead == 0);
            if (++s == nst) {
              s = 0;
              ph ^= 1;
            }
          }
          if (seg >= 1) mbar_wait(&tempty[as ^ 1], (((seg + 1) >> 1) - 1) & 1);
          tc_fence_after();
          for (int k = 0; k < ahead; ++k) {
            mma(s2, 1, acc2, k == 0);
            tc_commit_pair(&empty[s2]);
            if (++s2 == nst) s2 = 0;
          }
        }
        for (int kb = ahead; kb < num_kb; ++kb) {
          mbar_wait(&full[s], ph);
          tc_fence_after();
          mma(s, 0, acc, kb == 0);
          if (cnt == 2) mma(s, 1, acc2, false);
          tc_commit_pair(&empty[s]);
          if (++s == nst) {
            s = 0;
            ph ^= 1;
          }
        }
        tc_commit_pair(&tfull[as]);
        if (cnt == 2) tc_commit_pair(&tfull[as ^ 1]);
        seg += cnt;
      }
    }
    __syncwarp();
  } else {
    const int lg = warp & 3, quarter = (warp - 2) >> 2;
    const int et = threadIdx.x - 64;
    const bool scaled = KIND == KIND_I8 || ep.a_scale || ep.w_scale, by_two = epilogue_by_two(ep, EPI == EPI_LINEAR ? N : N >> 1);
    const bool ahead = EPI == EPI_LINEAR && ep.residual && by_two && !ep.out_f32;  // residuals are loaded before the accumulators are there
    griddep_wait();
    // this warp has read what it takes of an accumulator: the MMAs may write it again while the last chunk is finished
    auto give_back = [&](int as) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_relaxed(mapa_shared(smem_u32(&tempty[as]), 0));
    };
    int seg = 0, nt, mt, cnt;
    for (int unit = pair; unit < un.units; unit += pairs) {
      un.at(unit, nt, mt, cnt);
      const int n0w = nt * 2 * GEMM_BN + (int)rank * GEMM_BN + lg * 32;
      const int n = n0w + lane;
      for (int h = 0; h < cnt; ++h, ++seg) {
        const int as = seg & 1;
        const int m0 = (mt + h) * bt;
        named_bar_sync(1, 32 * PAIR_EPI_WARPS);  // the previous tile's readers of a_s_tile are done
        if (et < bt) a_s_tile[et] = (ep.a_scale && m0 + et < M) ? ep.a_scale[m0 + et] : 1.f;
        const float w_sc = (ep.w_scale && n < N) ? ep.w_scale[n] : 1.f;
        const float bias_v = (ep.bias && n < N) ? __bfloat162float(ep.bias[n]) : 0.f;
        named_bar_sync(1, 32 * PAIR_EPI_WARPS);
        uint32_t r[8] = {};
        int c0 = quarter * 16;
        if (ahead) epilogue_residual(ep, r, m0 + c0, M, n, N, lane & 1);
        mbar_wait(&tfull[as], (seg >> 1) & 1);
        __syncwarp();  // lanes may leave the wait one by one; tcgen05.ld wants them together
        tc_fence_after();
        const uint32_t acc = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(as * PAIR_MAX_BT);
        // the four warps of a lane group take every fourth chunk of 16 tokens
        uint32_t v[16];
        tmem_ld_32x32b_x16(acc + c0, v);  // bt >= 64: each of the four has a chunk
#pragma unroll 1
        for (; c0 < bt; c0 += 64) {
          tmem_ld_wait16(v);
          float f[16];
          uint32_t q[8];
#pragma unroll
          for (int j = 0; j < 16; ++j) f[j] = KIND == KIND_I8 ? (float)(int32_t)v[j] : __uint_as_float(v[j]);
#pragma unroll
          for (int j = 0; j < 8; ++j) q[j] = r[j];
          if (c0 + 64 < bt) {
            tmem_ld_32x32b_x16(acc + c0 + 64, v);
            if (ahead) epilogue_residual(ep, r, m0 + c0 + 64, M, n, N, lane & 1);
          } else {
            give_back(as);
          }
          epilogue_chunk_lanes<EPI>(ep, f, q, m0 + c0, M, n0w, N, lane, a_s_tile + c0, w_sc, bias_v, scaled, by_two);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // nobody leaves, or frees tensor memory, while the other CTA's MMAs or arrivals may still reach it
  if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * PAIR_MAX_BT);
}

namespace {

constexpr size_t PAIR_SMEM_RING = 232448 - 1024 - (PAIR_MAX_BT * 4 + 512);

int pair_stage_bytes(int bt, bool wide) { return (GEMM_BN + (wide ? bt : bt / 2)) * GEMM_BK_BYTES; }
int pair_stages(int stage) {
  int n = (int)(PAIR_SMEM_RING / (size_t)stage);
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
int launch_pair(const void* a, const void* w, const GemmEpilogue& ep, int M, int N, int K, int bt, int wide, cudaStream_t stream) {
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
  const int m_tiles = (M + bt - 1) / bt, n_tiles = (N + 2 * GEMM_BN - 1) / (2 * GEMM_BN), stage = pair_stage_bytes(bt, wide > 0);
  const PairUnits un(m_tiles, n_tiles, wide);
  const int used = un.units < pairs ? un.units : pairs;
  B200_CUDA_OK(launch_kernel_cluster(gemm_pair_kernel<KIND, EPI>, dim3(2 * used), dim3(PAIR_THREADS), PAIR_SMEM_RING + 1024, 2, stream, wm,
                                     am, ep, M, N, un, (K + BK - 1) / BK, bt, pair_stages(stage), stage, m_tiles == 1 ? 1 : 0));
  return B200_OK;
}

}  // namespace

void pair_shape(int M, int N, PairPlan p, int& units, int& stages, size_t& smem) {
  units = PairUnits((M + p.bt - 1) / p.bt, (N + 2 * GEMM_BN - 1) / (2 * GEMM_BN), p.wide).units;
  stages = pair_stages(pair_stage_bytes(p.bt, p.wide > 0));
  smem = PAIR_SMEM_RING + 1024;
}

// Tokens of a tile, and whether a pair takes two token tiles at once.  A wave of tiles costs its k-blocks -- 320 + 0.625 bt clocks each, the operands'
// way into shared memory and the MMAs' issue -- plus filling the ring, draining the last accumulator and the launch; so the widest tile wins unless
// a narrower one saves a wave or the padding of the last token tile.  Two at once cost 250 + 2.75 bt clocks a k-block, both accumulators' epilogue at the
// end and some of it between waves; the waves that would not fill go one by one where that ends sooner.  Fitted to and checked against 560 measured
// calls (bf16, fp8, SiLU and fp32 outputs, 129 to 4096 tokens, 14 weights, 11 to 17 plans each, L2 flushed): the choice is 0.6 % slower than the best
// plan on average, 14 % at most, and 0.966 of what the constants from before the MMAs were issued by an elected lane chose; 0.97 or less in 203
// calls, over 1.03 in four (1.05 at most).
// Measured (us, those constants / now, bf16): 777 x 6144 x 4096 50.0 / 39.2, 777 x 28672 x 4096 144 / 132, 2048 tokens of an fp8 prompt step 4265 / 4127.
PairPlan pair_plan(int M, int N, int K, int ab_dtype) {
  const int eb = ab_dtype == B200_BF16 ? 2 : 1, sms = sm_count();
  const int pairs = sms / 2, num_kb = (K * eb + GEMM_BK_BYTES - 1) / GEMM_BK_BYTES, n_tiles = (N + 2 * GEMM_BN - 1) / (2 * GEMM_BN);
  long long best_cost = 0;
  PairPlan best{0, 0};
  auto offer = [&](int bt, int wide, long long cost) {
    if (!best.bt || cost < best_cost) {
      best = PairPlan{bt, wide};
      best_cost = cost;
    }
  };
  for (int bt = PAIR_MAX_BT; bt >= 64; bt -= 32) {
    const int mt = (M + bt - 1) / bt;
    const long long lone_cost = (long long)num_kb * 5 * (512 + bt) / 8 + 4000 + 6 * bt;
    offer(bt, 0, ((long long)mt * n_tiles + pairs - 1) / pairs * lone_cost);
    if (mt < 2 || bt < 128) continue;
    const long long wide_cost = (long long)num_kb * (1000 + 11 * bt) / 4 + 2700 + 50 * bt, all = (long long)((mt + 1) / 2) * n_tiles;
    if (all > INT_MAX) continue;
    for (const long long wide : {all, all / pairs * pairs}) {  // wide to the end, or whole waves of it and the rest one by one
      if (!wide) continue;
      const PairUnits un(mt, n_tiles, (int)wide);
      const long long waves = (wide + pairs - 1) / pairs;
      offer(bt, (int)wide, waves * wide_cost + (waves - 1) * 2500 + (un.units - wide + pairs - 1) / pairs * lone_cost);
    }
  }
  return best;
}

// Whether a prompt-sized call stays with stream-K (gemm_tcgen05.cu), which cuts K: few tiles against a long K, or a nearly empty wave behind a full one.  Its
// time is about 25 us, 0.52 for each k-block of 128 x 256 of an SM's share and 8 for every CTA that adds to one tile; a wave of pairs stands here with the cost
// that it had while an MMA took 95 clocks to issue (640 clocks a k-block up to 128 tokens, from there 3 for each of the 128 + bt / 2 operand rows).  With
// today's costs the pairs would take more calls, up to 0.6 of the time, but they walk all of K in one accumulator, and the tensor cores cut the low bits
// of a sum at every 16 products, so a sum that stream-K cuts would lose more of them.  Measured, bf16, us and error of fp32 outputs against 64 bits, stream-K /
// pairs: 129 x 3584 x 18944 107 / 86, 0.36e-5 / 2.2e-5; 129 x 8192 x 28672 139 / 135, 1.2e-5 / 3.3e-5; 512 x 1024 x 28672 135 / 127, 0.32e-5 / 3.3e-5;
// 777 x 5120 x 27648 305 / 186, 2.3e-5 / 3.2e-5; fp8 4096 x 32000 x 2048 406 / 180, 7.05e-8 / 7.07e-8.
bool stream_k_keeps(int M, int N, int K, int ab_dtype) {
  const int eb = ab_dtype == B200_BF16 ? 2 : 1, sms = sm_count();
  const int pairs = sms / 2, num_kb = (K * eb + GEMM_BK_BYTES - 1) / GEMM_BK_BYTES, n_tiles = (N + 2 * GEMM_BN - 1) / (2 * GEMM_BN);
  long long pair_cost = LLONG_MAX;
  for (int bt = PAIR_MAX_BT; bt >= 64; bt -= 32) {
    const long long tiles = (long long)((M + bt - 1) / bt) * n_tiles, waves = (tiles + pairs - 1) / pairs;
    const long long cost = waves * ((long long)num_kb * (bt <= 128 ? 640 : 3 * (GEMM_BN + bt / 2)) + 2500 + 10 * bt);
    if (cost < pair_cost) pair_cost = cost;
  }
  const double sk_tiles = (double)((M + 255) / 256) * ((N + GEMM_BN - 1) / GEMM_BN), shared = sms / sk_tiles;
  const double stream_k_us = 25.0 + 0.52 * sk_tiles * num_kb / sms + 8.0 * (shared > 1.0 ? shared : 1.0);
  return stream_k_us * 1850.0 < (double)pair_cost;  // clocks at 1.85 GHz
}

// Decode-sized batches whose K the decode schedule does not cut (decode_on_pairs asks for that: bf16, fp8 and int8, 9 to 128 tokens, every epilogue but the
// rotating one).  A wave of pairs is bound by its k-blocks (0.247 us each) or by its weights (5.9 TB/s), behind 9.5 us of launch, first loads and epilogue; the
// decode schedule takes 12 us and 5.7 TB/s up to 64 tokens, 15 us and 5.0 TB/s above, where its tile of 128 tokens halves the ring.  The pairs have to
// win by a twentieth, above 64 tokens by 0.15.  Measured, us, decode schedule / pairs, L2 flushed: bf16 128 x 10272 x 2048 32.8 / 20.5, 64 x 55296 x 5120
// 119 / 101, 12 tokens 115 / 100, SiLU 128 139 / 102, 64 x 28672 x 4096 57.3 / 55.3, 128 fp32 63.5 / 57.3, 80 x 12288 x 4096 47.1 / 28.7; fp8 41 x 32000 x 2048
// 24.6 / 22.5, 128 x 28672 x 4096 SiLU 43.0 / 34.8; int8 64 x 49152 x 2048 38.9 / 28.7.  Over 492 such calls (20 weights, 12 to 128 tokens, linear, fp32 and
// SiLU outputs) none that goes to the pairs is slower there by more than 3 %.  Short rows as well: of 128 to 1536
// bytes, 4096 to 100000 of them, 0.96 of the time or less in 800 of 1080 calls.
bool pair_takes_decode(int M, int N, int K, int ab_dtype) {
  const long long row_bytes = (long long)K * (ab_dtype == B200_BF16 ? 2 : 1);
  const double row = (double)row_bytes, steps = 0.247 * ((row_bytes + GEMM_BK_BYTES - 1) / GEMM_BK_BYTES);
  const int pairs = sm_count() / 2, tiles = (N + 2 * GEMM_BN - 1) / (2 * GEMM_BN), rest = tiles % pairs;
  auto wave = [&](int n) {
    const double bytes = n * (2.0 * GEMM_BN) * row / 5.9e6;
    return n == 0 ? 0.0 : bytes > steps ? bytes : steps;
  };
  const double pair_us = 9.5 + (tiles / pairs) * wave(pairs) + wave(rest);
  return M <= 64 ? pair_us < 0.95 * (12.0 + N * row / 5.7e6) : pair_us < 0.85 * (15.0 + N * row / 5.0e6);
}

int launch_gemm_pair(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, int ab_dtype, PairPlan p,
                     cudaStream_t s) {
  if (ab_dtype == B200_BF16)
    return epi == EPI_SILU_MUL ? launch_pair<KIND_F16, EPI_SILU_MUL>(a, w, ep, M, N, K, p.bt, p.wide, s)
                               : launch_pair<KIND_F16, EPI_LINEAR>(a, w, ep, M, N, K, p.bt, p.wide, s);
  if (ab_dtype == B200_FP8_E4M3)
    return epi == EPI_SILU_MUL ? launch_pair<KIND_F8F6F4, EPI_SILU_MUL>(a, w, ep, M, N, K, p.bt, p.wide, s)
                               : launch_pair<KIND_F8F6F4, EPI_LINEAR>(a, w, ep, M, N, K, p.bt, p.wide, s);
  return epi == EPI_SILU_MUL ? launch_pair<KIND_I8, EPI_SILU_MUL>(a, w, ep, M, N, K, p.bt, p.wide, s)
                             : launch_pair<KIND_I8, EPI_LINEAR>(a, w, ep, M, N, K, p.bt, p.wide, s);
}

}  // namespace b200
