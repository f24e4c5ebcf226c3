// Expert GEMMs on CTA pairs (bf16 operands, fp32 sums): the rows of a step's (token, choice) pairs lie sorted by expert in row tiles, each
// owned by one expert, and how many tiles there are is known on the device only.
//   gate / up:  hid[row] = bf16(act(x W_gate^T, x W_up^T))        down:  out[pair of row] = hid W_down^T (fp32, scattered to pair order)
//
// The tile and the pipeline are gemm_pair.cu's: 256 weight rows x the row tile's tokens per pair of CTAs, tcgen05.mma.cta_group::2, two
// accumulators.  Prompt-sized batches (row tiles of 128): two neighbouring tiles of one expert run as one of 256 tokens, since a k-block
// costs a pair nearly the same either way.  Decode-sized ones (row tiles of 32): the weights of every expert that was chosen stream
// through the ring once, which is what bounds the step.  Gate / up: each CTA holds 64 gate rows and the 64 up rows of the same channels, so
// they meet in its shared memory: lanes that hold gates finish one half of a chunk's tokens, lanes that hold ups the other.
// Against the mma.sync kernels of moe.cu, 16 experts of 1024 on rows of 2048 (us): 8192 pairs, gate / up 244 -> 62
// and down 137 -> 35; 128 pairs 79 -> 31 and 32 -> 17, of which the weights take 20 and 10.
#include "gemm_group.cuh"
#include "gemm_pair.cuh"
#include "hybrid_common.cuh"

namespace b200 {

constexpr int GRP_MAX_TILES = 1024;  // row tiles whose schedule fits shared memory
constexpr int GRP_MAX_ST = 11;
constexpr int GRP_EPI_WARPS = 8;                      // two per 32-lane group of tensor memory: they share its token chunks
constexpr int GRP_THREADS = 64 + 32 * GRP_EPI_WARPS;  // + the TMA producer and the MMA issuer

template <bool GLU>
__global__ void __launch_bounds__(GRP_THREADS, 1)
    gemm_group_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map,
                      const __grid_constant__ CUtensorMap a2_map, const int32_t* __restrict__ sorted_ids,
                      const int32_t* __restrict__ tile_expert, const int32_t* __restrict__ num_tiles, int bm, int n_tiles, int num_kb, int nst,
                      int stage, void* __restrict__ out, int ldo, int outs, int scatter, float limit, int act) {
  constexpr int BK_ELEMS = GEMM_BK_BYTES / 2;
  constexpr int W_TILE = GEMM_BN * GEMM_BK_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[GRP_MAX_ST], empty[GRP_MAX_ST], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int32_t sched[GRP_MAX_TILES];  // first row tile << 17 | expert << 1 | (1: two tiles)
  __shared__ int32_t sched_n;
  // epilogue scratch, per half of the warps: GLU [2][16][64] exchanged values; then per warp a transposing tile
  __shared__ __align__(16) float xch[GLU ? 2 * 2 * 16 * 64 : 4];
  __shared__ __align__(16) float xpose[GLU ? GRP_EPI_WARPS * 16 * 20 : GRP_EPI_WARPS * XP_WARP_FLOATS];

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&w_map);
    tma_prefetch_desc(&a_map);
    tma_prefetch_desc(&a2_map);
    for (int s = 0; s < nst; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 2 * GRP_EPI_WARPS);
    }
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_slot, 2 * PAIR_MAX_BT);
    tmem_relinquish_pair();
  }
  griddep_launch();
  griddep_wait();  // the row tiles themselves are the predecessor's
  if (warp == 2) {
    // schedule: row tiles in order, neighbours of one expert two by two.  A run of one expert starts where its neighbour differs;
    // within the run, tiles at even distance from the start begin an entry.
    const int nt = min(*num_tiles, GRP_MAX_TILES);
    int count = 0, run = 0;  // run: first tile of the current expert's run (all lanes)
    int prev = -1;
    for (int base = 0; base < nt; base += 32) {
      const int t = base + lane;
      const int e = t < nt ? tile_expert[t] : -2;
      const int before = __shfl_up_sync(0xffffffffu, e, 1);
      const bool starts = e != (lane == 0 ? prev : before);
      int first = starts ? t : -1;  // start of this tile's run: the latest start at or before it
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, first, o);
        if (lane >= o && first < 0) first = v;
      }
      if (first < 0) first = run;
      const bool begins = t < nt && (bm < 128 || ((t - first) & 1) == 0);
      const int next = t + 1 < nt ? tile_expert[t + 1] : -2;
      const unsigned m = __ballot_sync(0xffffffffu, begins);
      if (begins) sched[count + __popc(m & ((1u << lane) - 1))] = (t << 17) | (e << 1) | (bm >= 128 && next == e ? 1 : 0);
      count += __popc(m);
      run = __shfl_sync(0xffffffffu, first, 31);
      prev = __shfl_sync(0xffffffffu, e, 31);
    }
    if (lane == 0) sched_n = count;
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const int tiles = sched_n * n_tiles;
  // rows of an expert's matrix per n-tile of a pair, and this CTA's part of them
  const int rows_e = GLU ? 2 * outs : outs;

  if (warp == 0) {
    if (elect_one()) {
      const uint64_t pol_w = policy_evict_first(), pol_a = policy_evict_last();
      int i = 0, s = 0, ph = 1;
      for (int tile = pair; tile < tiles; tile += pairs) {
        const int sc = sched[tile / n_tiles], n = tile % n_tiles;
        const int cnt = (sc & 1) ? 2 * bm : bm, e = (sc >> 1) & 0xffff;
        const int m0 = (sc >> 17) * bm + (int)rank * (cnt >> 1);
        const int w0 = e * rows_e + (GLU ? n * GEMM_BN + (int)rank * (GEMM_BN / 2) : n * 2 * GEMM_BN + (int)rank * GEMM_BN);
        const CUtensorMap* am = (sc & 1) ? &a2_map : &a_map;
        const uint32_t bytes = 2u * (uint32_t)(W_TILE + (cnt >> 1) * GEMM_BK_BYTES);
        for (int kb = 0; kb < num_kb; ++kb, ++i) {
          mbar_wait(&empty[s], ph);
          const uint32_t bar = mapa_shared(smem_u32(&full[s]), 0);
          uint8_t* ws = smem + (size_t)s * stage;
          if (rank == 0) mbar_expect_tx(&full[s], bytes);
          if constexpr (GLU) {
            tma_load_2d_pair(ws, &w_map, bar, kb * BK_ELEMS, w0, pol_w);
            tma_load_2d_pair(ws + W_TILE / 2, &w_map, bar, kb * BK_ELEMS, w0 + outs, pol_w);
          } else {
            tma_load_2d_pair(ws, &w_map, bar, kb * BK_ELEMS, w0, pol_w);
          }
          tma_load_2d_pair(ws + W_TILE, am, bar, kb * BK_ELEMS, m0, pol_a);
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
      int s = 0, ph = 0, seg = 0;
      for (int tile = pair; tile < tiles; tile += pairs, ++seg) {
        const int as = seg & 1, cnt = (sched[tile / n_tiles] & 1) ? 2 * bm : bm;
        const uint32_t idesc = umma_idesc(1, 1, 2 * GEMM_BN, (uint32_t)cnt);
        if (seg >= 2) mbar_wait(&tempty[as], ((seg >> 1) - 1) & 1);
        tc_fence_after();
        const uint32_t acc = tmem_base + (uint32_t)(as * PAIR_MAX_BT);
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(&full[s], ph);
          tc_fence_after();
          const uint32_t wa = smem_u32(smem + (size_t)s * stage), aa = wa + W_TILE;
#pragma unroll
          for (int kk = 0; kk < GEMM_BK_BYTES / 32; ++kk)
            umma_ss_pair<KIND_F16>(acc, umma_desc_sw128(wa + kk * 32), umma_desc_sw128(aa + kk * 32), idesc, (uint32_t)((kb | kk) != 0));
          tc_commit_pair(&empty[s]);
          if (++s == nst) {
            s = 0;
            ph ^= 1;
          }
        }
        tc_commit_pair(&tfull[as]);
      }
    }
    __syncwarp();
  } else {
    const int lg = warp & 3, half = (warp - 2) >> 2;
    int seg = 0;
    for (int tile = pair; tile < tiles; tile += pairs, ++seg) {
      const int as = seg & 1;
      const int sc = sched[tile / n_tiles], n = tile % n_tiles;
      const int cnt = (sc & 1) ? 2 * bm : bm, row0 = (sc >> 17) * bm;
      mbar_wait(&tfull[as], (seg >> 1) & 1);
      __syncwarp();  // lanes may leave the wait one by one; tcgen05.ld wants them together
      tc_fence_after();
      const uint32_t acc = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(as * PAIR_MAX_BT);
#pragma unroll 1
      for (int c0 = half * 32; c0 < cnt; c0 += 64) {
        uint32_t v0[16], v1[16];
        tmem_ld_32x32b_x16(acc + c0, v0);
        tmem_ld_32x32b_x16(acc + c0 + 16, v1);
        tmem_ld_wait();
        if constexpr (GLU) {
          // lanes of groups 0, 1: gates of channels 32 lg + lane, they finish tokens c0 .. c0 + 15; groups 2, 3: ups, tokens c0 + 16 ..
          const bool up = lg >= 2;
          const int ch = (lg & 1) * 32 + lane;
          float* mine = xch + half * (2 * 16 * 64) + (up ? 16 * 64 : 0) + ch;
          const float* theirs = xch + half * (2 * 16 * 64) + (up ? 0 : 16 * 64) + ch;
#pragma unroll
          for (int j = 0; j < 16; ++j) mine[j * 64] = __uint_as_float(up ? v0[j] : v1[j]);
          named_bar_sync(1 + half, 128);
          __nv_bfloat16* xb = reinterpret_cast<__nv_bfloat16*>(xpose + (warp - 2) * 16 * 20);  // [16 tokens][32 channels], pitch 40
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float o = theirs[j * 64];
            const float g = up ? o : __uint_as_float(v0[j]), u = up ? __uint_as_float(v1[j]) : o;
            xb[j * 40 + lane] = __float2bfloat16_rn(glu_act(g, u, act, limit));
          }
          __syncwarp();
          const int n0 = n * GEMM_BN + (int)rank * (GEMM_BN / 2) + (lg & 1) * 32;
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            const int mm = it * 8 + (lane >> 2), c8 = (lane & 3) * 8;
            const int row = row0 + c0 + (up ? 16 : 0) + mm;
            *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out) + (int64_t)row * ldo + n0 + c8) =
                *reinterpret_cast<const uint4*>(xb + mm * 40 + c8);
          }
          named_bar_sync(1 + half, 128);  // both tiles are rewritten by the next chunk
        } else {
          float* xp = xpose + (warp - 2) * XP_WARP_FLOATS;
          const int n0 = n * 2 * GEMM_BN + (int)rank * GEMM_BN + lg * 32;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int j = 0; j < 16; ++j) xp[j * XP_PITCH + lane] = __uint_as_float(q ? v1[j] : v0[j]);
            __syncwarp();
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              const int mm = it * 4 + (lane >> 3), c4 = (lane & 7) * 4;
              const int row = row0 + c0 + q * 16 + mm;
              const int id = sorted_ids[row];
              if (id >= 0)
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + (int64_t)(scatter ? id : row) * ldo + n0 + c4) =
                    *reinterpret_cast<const float4*>(xp + mm * XP_PITCH + c4);
            }
            __syncwarp();
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[as]), 0));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * PAIR_MAX_BT);
}

bool gemm_group_ok(const void* a, int lda, const void* w, int64_t w_stride, const void* out, int ldo, int row_tiles, int tile_rows, int N, int K,
                   bool glu) {
  return lda == K && K % 8 == 0 && N % (glu ? GEMM_BN : 2 * GEMM_BN) == 0 && w_stride == (int64_t)(glu ? 2 * N : N) * K && ldo % 8 == 0 &&
         row_tiles <= GRP_MAX_TILES && !((uintptr_t)a & 15) && !((uintptr_t)w & 15) && !((uintptr_t)out & 15) &&
         (tile_rows == 32 || tile_rows == 128);
}

template <bool GLU>
static int launch_group(const void* a, const int32_t* sorted_ids, const void* w, const int32_t* tile_expert, const int32_t* num_tiles,
                        int row_tiles, int tile_rows, int N, int K, void* out, int ldo, int scatter, float limit, int act, cudaStream_t st) {
  constexpr int BK = GEMM_BK_BYTES / 2;
  constexpr size_t RING = (GLU ? 192 : 202) * 1024;  // the rest holds the schedule and the epilogue's tiles
  auto kern = gemm_group_kernel<GLU>;
  B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(RING + 1024)));
  CUtensorMap wm, am, am2;
  // an expert's tiles never reach past its own rows (whole tiles only), so the map needs no edge below the last expert
  const int rows_box = GLU ? GEMM_BN / 2 : GEMM_BN;
  int rc = make_tmap_2d(&wm, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)1 << 31, (uint64_t)K * 2, BK, rows_box);
  if (rc) return rc;
  const uint64_t rows = (uint64_t)row_tiles * tile_rows;
  rc = make_tmap_2d(&am, a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, rows, (uint64_t)K * 2, BK, tile_rows / 2);
  if (rc) return rc;
  const int wide = tile_rows == 128 ? 256 : tile_rows;
  rc = make_tmap_2d(&am2, a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, rows, (uint64_t)K * 2, BK, wide / 2);
  if (rc) return rc;
  const int stage = GEMM_BN * GEMM_BK_BYTES + (wide / 2) * GEMM_BK_BYTES;
  int nst = (int)(RING / (size_t)stage);
  if (nst > GRP_MAX_ST) nst = GRP_MAX_ST;
  const int n_tiles = N / (GLU ? GEMM_BN : 2 * GEMM_BN);
  int pairs = sm_count() / 2;
  if ((long long)row_tiles * n_tiles < pairs) pairs = row_tiles * n_tiles;
  B200_CUDA_OK(launch_kernel_cluster(kern, dim3(2 * pairs), dim3(GRP_THREADS), RING + 1024, 2, st, wm, am, am2, sorted_ids, tile_expert,
                                     num_tiles, tile_rows, n_tiles, (K + BK - 1) / BK, nst, stage, out, ldo, N, scatter, limit, act));
  return B200_OK;
}

int launch_gemm_group(const void* a, const int32_t* sorted_ids, const void* w, const int32_t* tile_expert, const int32_t* num_tiles,
                      int row_tiles, int tile_rows, int N, int K, void* out, int ldo, int scatter, bool glu, float limit, int act,
                      cudaStream_t st) {
  return glu ? launch_group<true>(a, sorted_ids, w, tile_expert, num_tiles, row_tiles, tile_rows, N, K, out, ldo, scatter, limit, act, st)
             : launch_group<false>(a, sorted_ids, w, tile_expert, num_tiles, row_tiles, tile_rows, N, K, out, ldo, scatter, limit, act, st);
}

}  // namespace b200
