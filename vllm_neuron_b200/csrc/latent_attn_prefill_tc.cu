// Attention over cached latents, prompt portions (bf16 pools, pages of 32 tokens): one pool holds keys and values -- a token's row is
// [normed latent (C columns) | rotated key part], the scores take the whole row, the values are its first C columns, all heads share it.
// Capability of the reference's latent-attention layers: exploded.py (prefill) -- there a dense attention over the up-projected keys.
//
// A CTA owns 128 query tokens of one head and walks the keys it sees in steps of 64 (two pages).  The step's rows come ONCE, by TMA, as
// columns of 64 (128-byte swizzle): as they lie they are the K-major operand of S = Q K^T and, their first C columns, the MN-major operand
// of O += P V.  S is double buffered in tensor memory (the scores of step j + 1 are there while step j is weighted), the weights go back over
// their scores as bf16, O stays in C columns of tensor memory and is scaled only when a row's maximum grew by more than 2^8.
// The weights go as two bf16 terms: with one, and a maximum that moves in steps, the difference from 64 bits was 5 % above that of the mma.sync
// kernel which these portions took before (3.19e-3 / 3.03e-3 relative, now 2.93e-3).
// What bounds it: the products of a step, 20 score MMAs of 6 KB of operands from shared memory at 320 columns (~950 clocks) and 8 of the values
// (512), then a step's weights on the way (1100 clocks, beside the next scores).  16 heads, rows of 320, 1600 tokens: 310 us on mma.sync, here 51; 16 tokens
// at 1800 227 / 45.  Before all threads laid down the queries and the output went through shared memory 96, before the elected lane 63.
// Steps of 64 keys: 80 KB of queries and three stages of 40 KB fill the shared memory at 320 columns; 128 keys would leave one stage.
// Rows of up to 192 columns: two stages, so that two CTAs share an SM.
#include "common.cuh"
#include "gemm_common.cuh"

namespace b200 {

int kv_pool_tmap(const void* pool, int num_blocks, int Hkv, int D, CUtensorMap* out);  // boxes of 64 columns x 32 rows, 128B swizzle

constexpr int LP_BM = 128;        // query tokens of a tile
constexpr int LP_BN = 64;         // keys of a step
constexpr int LP_BLK = 32;        // tokens per page
constexpr int LP_THREADS = 256;   // warps 0-3 weights, 4 MMA, 5 and 6 load a page of a step each
constexpr int LP_QCH = LP_BM * 128, LP_KCH = LP_BN * 128;  // 64 columns of the query tile / of a step's keys

// C: value columns; rows of D = 16 n columns, C <= D <= C + 64.  ST: stages of keys.
template <int C, int ST>
__global__ void __launch_bounds__(LP_THREADS, C <= 128 ? 2 : 1)
    latent_prefill_tc_kernel(const __grid_constant__ CUtensorMap k_map, const float* __restrict__ q, int ldq,
                             const int32_t* __restrict__ block_table, int64_t bt_stride, const int32_t* __restrict__ seq_start,
                             const int32_t* __restrict__ seq_slot, const int32_t* __restrict__ seq_pos0,
                             __nv_bfloat16* __restrict__ out, int H, int D, float scale, int window, const float* __restrict__ sink) {
  constexpr int CH = C / 64 + 1;  // pieces of 64 columns: the values' and the rest of the row (columns past D come as zeros)
  constexpr int KST = CH * LP_KCH;
  constexpr uint32_t TMEM_COLS = C <= 128 ? 256 : 512;
  constexpr uint32_t O_COL = 2 * LP_BN;
  constexpr uint32_t IDESC_S = umma_idesc(1, 1, LP_BM, LP_BN);
  constexpr uint32_t IDESC_PV = umma_idesc(1, 1, LP_BM, C) | (1u << 16);  // B (= V) is MN-major

  const int sq = blockIdx.z, head = blockIdx.x;
  const int t0 = seq_start[sq], n_new = seq_start[sq + 1] - t0;
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * LP_BM;  // a causal tile's cost grows with its index: the last ones first
  if (q0 >= n_new) return;
  const int pos0 = seq_pos0[sq];
  const int32_t* bt_row = block_table + (int64_t)seq_slot[sq] * bt_stride;
  const int q_hi = min(q0 + LP_BM, n_new);
  const int kv_end = pos0 + q_hi;  // keys [0, kv_end) are visible to some row of the tile
  auto first_key = [&](int pos) { return pos >= window ? pos - window + 1 : 0; };
  const int j_lo = first_key(pos0 + q0) / LP_BN;
  const int niter = (kv_end + LP_BN - 1) / LP_BN - j_lo;
  const int nblk = (kv_end + LP_BLK - 1) / LP_BLK;  // pages that hold these keys

  extern __shared__ uint8_t smem_raw[];
  uint8_t* q_s = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* k_s = q_s + CH * LP_QCH;  // [ST][CH][64 keys][128 B]
  uint64_t* k_full = reinterpret_cast<uint64_t*>(k_s + ST * KST);  // ST
  uint64_t* k_empty = k_full + ST;   // ST
  uint64_t* s_full = k_empty + ST;   // 2
  uint64_t* p_ready = s_full + 2;    // 2 x 2 (buffer, half of the step's keys)
  uint64_t* o_done = p_ready + 4;    // 1: the products of a step
  uint64_t* o_full = o_done + 1;     // 1: those of all steps (a waiter may be two steps behind o_done here, which its parity cannot tell)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (warp == 4) {
    if (lane == 0) {
      tma_prefetch_desc(&k_map);
      for (int s = 0; s < ST; ++s) mbar_init(&k_full[s], 2), mbar_init(&k_empty[s], 1);
      for (int b = 0; b < 2; ++b) mbar_init(&s_full[b], 1), mbar_init(&p_ready[2 * b], 4), mbar_init(&p_ready[2 * b + 1], 4);
      mbar_init(o_done, 1);
      mbar_init(o_full, 1);
      fence_mbar_init();
      fence_proxy_async();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  griddep_launch();
  griddep_wait();  // q and the pool were written by the previous kernels of the stream
  const uint32_t tmem = *tmem_slot;

  // keys, page `warp - 5` of step it (warps 5 and 6, one lane)
  auto load_keys = [&](int it) {
    const int half = warp - 5, s = it % ST, bi = (j_lo + it) * 2 + half;
    const int blk = bi < nblk ? __ldg(bt_row + bi) : 0;  // past the keys: the null page (masked, and laid to zero as values)
    if (it >= ST) mbar_wait(&k_empty[s], (uint32_t)(it / ST - 1) & 1u);
    mbar_expect_tx(&k_full[s], (uint32_t)KST / 2);
    uint8_t* dst = k_s + s * KST + half * (LP_BLK * 128);
#pragma unroll
    for (int c = 0; c < CH; ++c) tma_load_2d(dst + c * LP_KCH, &k_map, &k_full[s], c * 64, blk * LP_BLK);
  };
  if ((warp == 5 || warp == 6) && elect_one())
    for (int it = 0; it < min(ST, niter); ++it) load_keys(it);
  __syncwarp();
  // q tile, all threads: fp32 rows -> bf16, K-major 128B swizzle; four pieces of 8 columns in flight a thread (128 rows of 320: 20 pieces each)
  {
    const float* qsrc = q + (int64_t)(t0 + q0) * ldq + (int64_t)head * D;
    const int pieces = D >> 3, n = D >> 4, drow = LP_THREADS / pieces, dc = LP_THREADS - drow * pieces;
    int row = threadIdx.x / pieces, c = threadIdx.x - row * pieces;
    for (int i0 = 0; i0 < n; i0 += 4) {
      float4 a[4], b[4];
      int off[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        off[k] = (c >> 3) * LP_QCH + row * 128 + (((c & 7) ^ (row & 7)) << 4);
        a[k] = b[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i0 + k < n && q0 + row < n_new) {
          const float* src = qsrc + (int64_t)row * ldq + c * 8;
          a[k] = *reinterpret_cast<const float4*>(src), b[k] = *reinterpret_cast<const float4*>(src + 4);
        }
        row += drow, c += dc;
        if (c >= pieces) c -= pieces, ++row;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i0 + k < n)
          *reinterpret_cast<uint4*>(q_s + off[k]) =
              make_uint4(pack_bf16(a[k].x, a[k].y), pack_bf16(a[k].z, a[k].w), pack_bf16(b[k].x, b[k].y), pack_bf16(b[k].z, b[k].w));
    }
    fence_proxy_async();  // the tensor core reads these bytes through the async proxy
    __syncthreads();
  }

  if (warp == 5 || warp == 6) {
    if (elect_one())
      for (int it = ST; it < niter; ++it) load_keys(it);
    __syncwarp();
  } else if (warp == 4) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {  // (an elected lane: the operands of an MMA stay in uniform registers; by lane == 0 an issue takes twice as long)
      const int steps = D / 16;
      auto issue_s = [&](int it) {
        const int s = it % ST;
        mbar_wait(&k_full[s], (uint32_t)(it / ST) & 1u);
        tc_fence_after();
        const uint32_t qa = smem_u32(q_s), ka = smem_u32(k_s + s * KST), d = tmem + (uint32_t)(it & 1) * LP_BN;
        for (int kk = 0; kk < steps; ++kk)
          umma_ss<KIND_F16>(d, umma_desc_sw128(qa + (uint32_t)(kk >> 2) * LP_QCH + (uint32_t)(kk & 3) * 32),
                            umma_desc_sw128(ka + (uint32_t)(kk >> 2) * LP_KCH + (uint32_t)(kk & 3) * 32), IDESC_S, (uint32_t)(kk != 0));
        tc_commit(&s_full[it & 1]);
      };
      issue_s(0);
      if (niter > 1) issue_s(1);
      for (int it = 0; it < niter; ++it) {
        const int s = it % ST;
        const uint32_t va = smem_u32(k_s + s * KST), p = tmem + (uint32_t)(it & 1) * LP_BN;
#pragma unroll
        for (int kk = 0; kk < LP_BN / 16; ++kk) {  // 16 keys: two 8-row groups of the [key][column] pieces
          if ((kk & 1) == 0) {
            mbar_wait(&p_ready[2 * (it & 1) + (kk >> 1)], (uint32_t)(it >> 1) & 1u);
            tc_fence_after();
          }
          const uint64_t vd = umma_desc_mn_sw128(va + kk * 2048, LP_KCH, 1024);
          umma_ts_f16(tmem + O_COL, p + (uint32_t)kk * 8u, vd, IDESC_PV, (uint32_t)((it | kk) != 0));
          umma_ts_f16(tmem + O_COL, p + 32u + (uint32_t)kk * 8u, vd, IDESC_PV, 1u);
        }
        tc_commit(&k_empty[s]);
        tc_commit(o_done);
        if (it + 2 < niter) issue_s(it + 2);  // over the weights of step `it`: the products that read them were issued before
      }
      tc_commit(o_full);
    }
    __syncwarp();
  } else if (warp < 4) {
    // ------------------------------------------------------------------ weights, one row per thread
    const int row = threadIdx.x;
    const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
    const uint32_t o_addr = lanes + O_COL;
    const int qpos = pos0 + q0 + row;
    const int klo = first_key(qpos), klo_first = first_key(pos0 + q0), klo_last = first_key(pos0 + q0 + LP_BM - 1);
    constexpr float LOG2E = 1.4426950408889634f;
    const float sl = scale * LOG2E;
    // a sink is a key without a value: the running maximum starts at its logit (not scaled), the denominator at its 1
    float m_used = sink ? sink[head] * LOG2E : -INFINITY, l = sink ? 1.f : 0.f;
    for (int it = 0; it < niter; ++it) {
      const uint32_t s_addr = lanes + (uint32_t)(it & 1) * LP_BN;
      const int k0 = (j_lo + it) * LP_BN;
      const bool masked = k0 + LP_BN - 1 > pos0 + q0 || k0 < klo_last;  // some key of the step is hidden from some row
      mbar_wait(&s_full[it & 1], (uint32_t)(it >> 1) & 1u);
      tc_fence_after();
      uint32_t sv[LP_BN];
      tmem_ld_32x32b_x32(s_addr, &sv[0]);
      tmem_ld_32x32b_x32(s_addr + 32, &sv[32]);
      tmem_ld_wait();
      if (masked) {
#pragma unroll
        for (int i = 0; i < LP_BN; ++i)
          if (k0 + i > qpos || k0 + i < klo) sv[i] = 0xff800000u;
        // keys that no row of the tile sees -- past the tile's last, ahead of the first row's window -- are values with weight 0: whatever their pages hold
        // there must be finite
        const int head = klo_first - k0, tail = kv_end - k0;  // the step's seen keys are head .. tail - 1
        if (head > 0 || tail < LP_BN) {
          uint8_t* ks = k_s + (it % ST) * KST;
          for (int idx = row; idx < (C / 64) * LP_BN * 8; idx += 128) {
            const int c = idx / (LP_BN * 8), r = idx - c * (LP_BN * 8), key = r >> 3;
            if (key < head || key >= tail) *reinterpret_cast<uint4*>(ks + c * LP_KCH + r * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async();
        }
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < LP_BN; i += 8) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mx4[k] = fmaxf(mx4[k], fmaxf(__uint_as_float(sv[i + 2 * k]), __uint_as_float(sv[i + 2 * k + 1])));
      }
      const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl);
      // lazy maximum: move it (and pay the O read-modify-write) only when it grew by more than 2^8
      const bool grow = m_new > m_used + 8.f;
      if (__any_sync(0xffffffffu, grow)) {
        const float alpha = grow ? ex2_approx(m_used - m_new) : 1.f;  // m_used = -inf -> 0
        if (grow) m_used = m_new;
        l *= alpha;
        if (it > 0) {
          mbar_wait(o_done, (uint32_t)(it - 1) & 1u);
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < C / 32; ++c) {
            uint32_t v[32];
            tmem_ld_32x32b_x32(o_addr + c * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            tmem_st_32x32b_x32(o_addr + c * 32, v);
          }
          tmem_st_wait();
        }
      }
      const float neg_m = m_used == -INFINITY ? 0.f : -m_used;  // a row that has seen no key yet: 2^(-inf) = 0, not NaN
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < LP_BN / 32; ++c) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = ex2_approx(fmaf(__uint_as_float(sv[c * 32 + i]), sl, neg_m));
          const float p1 = ex2_approx(fmaf(__uint_as_float(sv[c * 32 + i + 1]), sl, neg_m));
          l4[(i >> 1) & 3] += p0 + p1;
          const uint32_t h = pack_bf16(p0, p1);
          hi[i >> 1] = h;
          lo[i >> 1] = pack_bf16(p0 - __uint_as_float(h << 16), p1 - __uint_as_float(h & 0xffff0000u));
        }
        tmem_st_32x32b_x16(s_addr + c * 16, hi);
        tmem_st_32x32b_x16(s_addr + 32 + c * 16, lo);
        tmem_st_wait();  // the products of the first 32 keys run while the other weights are made (512 tokens at 4000, 16 heads of 320: 98.4 -> 95.5 us)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[2 * (it & 1) + c]);
      }
      l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
    }
    // ------------------------------------------------------------------ O / l -> rows of the output
    mbar_wait(o_full, 0);
    tc_fence_after();
    const float inv = l > 0.f ? 1.f / l : 0.f;
    // a row per thread in, rows of 2 C bytes out, through the warp's part of the key stages (every product has read them): 16-byte piece p of row r
    // sits at piece p ^ (r % 8)
    uint8_t* ws = k_s + warp * (32 * C * 2);
#pragma unroll 1
    for (int c = 0; c < C / 32; ++c) {
      uint32_t v[32];
      tmem_ld_32x32b_x32(o_addr + c * 32, v);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; i += 8)
        *reinterpret_cast<uint4*>(ws + lane * (C * 2) + (((c * 4 + (i >> 3)) ^ (lane & 7)) << 4)) =
            make_uint4(pack_bf16(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv),
                       pack_bf16(__uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv),
                       pack_bf16(__uint_as_float(v[i + 4]) * inv, __uint_as_float(v[i + 5]) * inv),
                       pack_bf16(__uint_as_float(v[i + 6]) * inv, __uint_as_float(v[i + 7]) * inv));
    }
    __syncwarp();
    constexpr int PR = C / 8, RW = 32 / PR;  // pieces of a row, rows a store of the warp takes
    const int r0 = warp * 32, rows = min(32, q_hi - q0 - r0), lr = lane / PR, lp = lane % PR;
    __nv_bfloat16* dst = out + ((int64_t)(t0 + q0 + r0) * H + head) * C + lp * 8;
#pragma unroll 8
    for (int r = lr; r < rows; r += RW)
      *reinterpret_cast<uint4*>(dst + (int64_t)r * H * C) = *reinterpret_cast<const uint4*>(ws + r * (C * 2) + ((lp ^ (r & 7)) << 4));
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) tmem_dealloc(tmem, TMEM_COLS);
}

template <int C, int ST>
static int lp_launch(const CUtensorMap& km, const float* q, int ldq, const int32_t* block_table, int64_t bt_stride, const int32_t* seq_start,
                     const int32_t* seq_slot, const int32_t* seq_pos0, int B, int max_new, void* out, int H, int D, float scale, int window,
                     const float* sink, cudaStream_t stream) {
  auto kern = latent_prefill_tc_kernel<C, ST>;
  const size_t smem = (size_t)(C / 64 + 1) * (LP_QCH + ST * LP_KCH) + 256 + 1024;
  static bool attr_done = false;
  if (!attr_done) {
    B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_done = true;
  }
  B200_CUDA_OK(launch_kernel(kern, dim3(H, (max_new + LP_BM - 1) / LP_BM, B), dim3(LP_THREADS), smem, stream, km, q, ldq, block_table, bt_stride,
                             seq_start, seq_slot, seq_pos0, reinterpret_cast<__nv_bfloat16*>(out), H, D, scale, window, sink));
  return B200_OK;
}

}  // namespace b200

using namespace b200;

extern "C" {

// 1 when b200_latent_attn_prefill_tc has a kernel for rows of D columns with C value columns
int b200_latent_attn_prefill_tc_supported(int D, int C, int block_size) {
  return block_size == LP_BLK && (C == 128 || C == 256) && D >= C && D <= C + 64 && D % 16 == 0;
}

int b200_latent_attn_prefill_tc(const float* q, int ldq, const void* pool, int num_blocks, const int32_t* block_table, int64_t bt_stride,
                                const int32_t* seq_start, const int32_t* seq_slot, const int32_t* seq_pos0, int B, int max_new,
                                const float* sink, float scale, int window, void* out, int H, int D, int C, int block_size, void* stream) {
  B200_REQUIRE(window >= 1, "latent_attn_prefill_tc: window %d", window);
  B200_REQUIRE(q && pool && block_table && seq_start && seq_slot && seq_pos0 && out, "latent_attn_prefill_tc: null pointer");
  B200_REQUIRE(H > 0, "latent_attn_prefill_tc: %d query heads", H);
  if (!b200_latent_attn_prefill_tc_supported(D, C, block_size) || !(scale > 0.f) || (ldq & 3) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15)) {
    set_last_error("latent_attn_prefill_tc: rows of %d columns with %d values, a scale of %g or the layout of q have no kernel", D, C, (double)scale);
    return B200_ERR_UNSUPPORTED;
  }
  if (B <= 0 || max_new <= 0) return B200_OK;
  CUtensorMap km;
  int rc = kv_pool_tmap(pool, num_blocks, 1, D, &km);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  if (C == 256)
    return lp_launch<256, 3>(km, q, ldq, block_table, bt_stride, seq_start, seq_slot, seq_pos0, B, max_new, out, H, D, scale, window, sink, st);
  return lp_launch<128, 2>(km, q, ldq, block_table, bt_stride, seq_start, seq_slot, seq_pos0, B, max_new, out, H, D, scale, window, sink, st);
}

}  // extern "C"
