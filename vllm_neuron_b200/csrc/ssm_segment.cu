// Segments of the state-space scan (ssm_scan.cu) as matrix products: bf16 x, B, C, fp32 everything else.
//
// Inside a segment of at most 128 tokens, with cum_i the sum of the log decays up to token i and S_in the state before the segment,
//   y_i   = exp(cum_i) S_in C_i  +  sum_{j <= i} (C_i . B_j) exp(cum_i - cum_j) dt_j x_j  +  D x_i
//   S_out = exp(cum_end) S_in    +  sum_j exp(cum_end - cum_j) dt_j x_j B_j^T
// which is the recurrence with its sums regrouped.  One operand of every product is exact in bf16 (x, B or C); the other (the weighted
// scores, the state, the weighted x) is fp32 and enters as THREE bf16 terms that together hold its 24 mantissa bits, so products are
// exact; their sums, 16 tokens or state elements at a time, are the tensor cores' (below).  The cumulated log decays are summed in 64 bits and kept as a pair of floats: the
// difference of two of them is good to fp32 wherever in the segment it is taken.
//
// Why: the sequential kernel walks tokens at ~0.19 us each (two passes over a segmented portion) and issues 5 fp32 operations per state
// element and token on the FMA pipe; mma.sync does the regrouped sums, three terms included, in a seventh of the issue slots.  Per
// (head, segment) the output kernel runs 5 400 m16n8k16 products (about 6 us of tensor pipe) on 160 KB of operands, one CTA per SM: load,
// split and products follow one another, which is what bounds it now (18 us).  One portion of 4096 tokens, 32 heads of 128 x 128: 843 us
// sequential, 217 us here; the outputs are more than half of it.
#include "ssm_common.cuh"

namespace b200 {

constexpr int SEG_THREADS = 256;
constexpr int SEG_OUT_THREADS = 512;

// fp32 -> three bf16 terms (round to nearest each): v = h + m + l up to 2^-25 |v|
__device__ __forceinline__ void split3(float2 v, uint32_t& h, uint32_t& m, uint32_t& l) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y);
  const float2 r = make_float2(v.x - __low2float(a), v.y - __high2float(a));
  const __nv_bfloat162 b = __floats2bfloat162_rn(r.x, r.y);
  const __nv_bfloat162 c = __floats2bfloat162_rn(r.x - __low2float(b), r.y - __high2float(b));
  h = *reinterpret_cast<const uint32_t*>(&a);
  m = *reinterpret_cast<const uint32_t*>(&b);
  l = *reinterpret_cast<const uint32_t*>(&c);
}

// The tensor cores cut a sum's low bits where the CUDA cores round; longer sums are therefore made of fresh MMA results -- one for 16 exact
// products, three in a chain where an operand has its three terms -- with rounded additions.  Against 64 bits (2-norm of the difference
// over that of the result, 4096 and 8192 tokens; sequential kernel in brackets): step sizes of a tenth and more: outputs 0.9 - 1.0e-7 (0.8 -
// 0.97e-7), states 0.5 - 0.9e-7 (0.5 - 0.98e-7); of a few thousandths: outputs 0.7 - 0.98e-7 (3.8 - 6.5e-7), states 1.0 - 1.1e-7 (4.1 -
// 9.0e-7); of a few ten-thousandths: outputs 1.1 - 1.5e-7 (1.0 - 6.9e-6), states 1.9 - 3.0e-7 (1.9 - 17e-6).
__device__ __forceinline__ void add_to(float (&a)[4], const float (&b)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] += b[i];
}

// step sizes and cumulated log decays of the segment's tokens (zero step past its end): dts[i], cum[i] = (high, low) floats.
// All threads; ends with a barrier.  Returns the sum of the step sizes to thread 127.
__device__ __forceinline__ float segment_decays(const float* __restrict__ dt_in, int ld_dt, int dt_col, int t0, int n, float negA,
                                                float bias, float* dts, float2* cum, double* part) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double v = 0.0, s = 0.0;
  if (tid < SEG_TOKENS) {
    float dt = 0.f;
    if (tid < n) {
      const float z = dt_in[(int64_t)(t0 + tid) * ld_dt + dt_col] + bias;
      dt = z > 20.f ? z : log1pf(expf(z));  // softplus, no clamp on the step size
    }
    dts[tid] = dt;
    v = (double)dt;
    s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    if (lane == 31) part[warp] = s;
  }
  __syncthreads();
  if (tid < SEG_TOKENS) {
    for (int w = 0; w < warp; ++w) s += part[w];
    const double c = (double)negA * s;
    const float hi = (float)c;
    cum[tid] = make_float2(hi, (float)(c - (double)hi));
  }
  __syncthreads();
  return (float)s;
}

__device__ __forceinline__ int nonfinite_bf16x2(uint32_t v) { return (v & 0x7f80u) == 0x7f80u || (v & 0x7f800000u) == 0x7f800000u; }

// rows [t0, t0 + n) x COLS bf16 columns from col -> smem rows of COLS + 8; rows past n are zeros
template <int COLS, int THREADS>
__device__ __forceinline__ void load_rows(const __nv_bfloat16* __restrict__ src, int ld, int64_t col, int t0, int n, __nv_bfloat16* dst) {
  constexpr int PIECES = COLS / 8;
  for (int i = threadIdx.x; i < SEG_TOKENS * PIECES; i += THREADS) {
    const int r = i / PIECES, c = (i % PIECES) * 8;
    cp_async16(smem_u32(dst + r * (COLS + 8) + c), src + (int64_t)(t0 + (r < n ? r : 0)) * ld + col + c, r < n);
  }
}

// What the products below cannot do -- infinite or NaN x, which a masked weight of zero would carry into the earlier tokens of its block, and
// segments of more tokens, which no caller cuts for this form: the recurrence as it stands, a value column per thread.
template <int P, int N, bool OUT>
__device__ __noinline__ void walk_segment(const __nv_bfloat16* __restrict__ xbc, int C, const float* __restrict__ dt_in, int ld_dt, int dt_col,
                                          int t0, int n, int64_t xcol, int64_t bcol, int64_t ccol, float negA, float bias, float dsk,
                                          const float* __restrict__ S_in, float* __restrict__ S_out, float* __restrict__ y, int ldy,
                                          float* __restrict__ dtsum) {
  const int p = threadIdx.x;
  if (p >= P) return;
  float S[N], total = 0.f;
  for (int k = 0; k < N; ++k) S[k] = S_in ? S_in[p * N + k] : 0.f;
  for (int t = t0; t < t0 + n; ++t) {
    const float z = dt_in[(int64_t)t * ld_dt + dt_col] + bias;
    const float dt = z > 20.f ? z : log1pf(expf(z)), dec = expf(negA * dt);
    const __nv_bfloat16* row = xbc + (int64_t)t * C;
    const float x = __bfloat162float(row[xcol + p]);
    float acc = 0.f;
    for (int k = 0; k < N; ++k) {
      S[k] = dec * S[k] + __bfloat162float(row[bcol + k]) * (dt * x);
      if (OUT) acc += S[k] * __bfloat162float(row[ccol + k]);
    }
    if (OUT) y[(int64_t)t * ldy + xcol + p] = acc + dsk * x;
    total += dt;
  }
  if (!OUT) {
    for (int k = 0; k < N; ++k) S_out[p * N + k] = S[k];
    if (p == 0) *dtsum = total;
  }
}

// S_loc[p][n] = sum_j exp(cum_end - cum_j) dt_j x_j[p] B_j[n] of one (head, segment) -> scratch entry segment + 1, where the chaining pass
// makes the next segment's start state of it; of a sequence's last segment -> its first entry, which no start state needs (the first segment
// starts from the slot).  Also the segment's summed step size.  8 warps as P / 32 x 8 / (P / 32) tiles of 32 value columns.
template <int P, int N>
__global__ void __launch_bounds__(SEG_THREADS, 2)
    ssd_segment_state_kernel(const __nv_bfloat16* __restrict__ xbc, int C, const float* __restrict__ dt_in, int ld_dt, int dt_col0,
                             const float* __restrict__ A_log, const float* __restrict__ dt_bias, int H, int G, const int4* __restrict__ segs,
                             const int32_t* __restrict__ seq_seg0, float* __restrict__ seg_state, float* __restrict__ seg_dtsum) {
  griddep_launch();
  griddep_wait();
  constexpr int WP = P / 32, WN = 8 / WP, NT = N / WN / 8;  // n8 tiles per warp
  extern __shared__ __align__(16) unsigned char seg_smem[];
  __nv_bfloat16* Xs = reinterpret_cast<__nv_bfloat16*>(seg_smem);  // [128][P + 8]
  __nv_bfloat16* Bs = Xs + SEG_TOKENS * (P + 8);                   // [128][N + 8]
  __shared__ float dts[SEG_TOKENS];
  __shared__ float2 cum[SEG_TOKENS];
  __shared__ double part[4];
  const int4 sd = segs[blockIdx.y];
  const int t0 = sd.x, n = sd.y - sd.x, h = blockIdx.x;
  if (seg_is_short(sd)) return;
  const int64_t bcol = (int64_t)H * P + (int64_t)(h / (H / G)) * N;
  const int entry = (sd.w & SEG_LAST) ? seq_seg0[sd.z] : (int)blockIdx.y + 1;
  float* dst = seg_state + ((int64_t)entry * H + h) * (P * N);
  if (n > SEG_TOKENS) {
    walk_segment<P, N, false>(xbc, C, dt_in, ld_dt, dt_col0 + h, t0, n, (int64_t)h * P, bcol, 0, -expf(A_log[h]), dt_bias[h], 0.f, nullptr, dst,
                              nullptr, 0, seg_dtsum + (int64_t)blockIdx.y * H + h);
    return;
  }
  load_rows<P, SEG_THREADS>(xbc, C, (int64_t)h * P, t0, n, Xs);
  load_rows<N, SEG_THREADS>(xbc, C, bcol, t0, n, Bs);
  cp_async_commit();
  const float total = segment_decays(dt_in, ld_dt, dt_col0 + h, t0, n, -expf(A_log[h]), dt_bias[h], dts, cum, part);
  if (threadIdx.x == SEG_TOKENS - 1) seg_dtsum[(int64_t)blockIdx.y * H + h] = total;
  if (threadIdx.x < SEG_TOKENS) {  // dts becomes the token's weight at the segment's end
    const float2 end = cum[SEG_TOKENS - 1], c = cum[threadIdx.x];
    dts[threadIdx.x] *= expf((end.x - c.x) + (end.y - c.y));
  }
  cp_async_wait<0>();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p0 = (warp / WN) * 32, n0 = (warp % WN) * (N / WN);
  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;
  const int ksteps = (n + 15) / 16;
  for (int k = 0; k < ksteps; ++k) {
    const int tk = k * 16 + 2 * (lane & 3);
    const float2 w0 = make_float2(dts[tk], dts[tk + 1]), w1 = make_float2(dts[tk + 8], dts[tk + 9]);
    uint32_t ah[2][4], am[2][4], al[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t x[4];
      ldmatrix_x4_trans(x, smem_u32(Xs + (k * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * (P + 8) + p0 + i * 16 + ((lane >> 3) & 1) * 8));
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[r]));
        const float2 w = r < 2 ? w0 : w1;
        split3(make_float2(v.x * w.x, v.y * w.y), ah[i][r], am[i][r], al[i][r]);
      }
    }
#pragma unroll
    for (int jj = 0; jj < NT / 2; ++jj) {
      uint32_t b[4];
      ldmatrix_x4_trans(b, smem_u32(Bs + (k * 16 + (lane & 15)) * (N + 8) + n0 + jj * 16 + (lane >> 4) * 8));
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float t[4] = {};
          mma_bf16_16816(t, al[i], b[2 * u], b[2 * u + 1]);
          mma_bf16_16816(t, am[i], b[2 * u], b[2 * u + 1]);
          mma_bf16_16816(t, ah[i], b[2 * u], b[2 * u + 1]);
          add_to(acc[i][2 * jj + u], t);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        *reinterpret_cast<float2*>(dst + (p0 + i * 16 + (lane >> 2) + 8 * r) * N + n0 + j * 8 + 2 * (lane & 3)) =
            make_float2(acc[i][j][2 * r], acc[i][j][2 * r + 1]);
}

// y of one (head, segment) from the segment's start state.  A warp owns 16 tokens x half of the columns (the scores are computed twice,
// a tenth of the products, for twice the warps to hide them); token blocks are dealt so that the four warps of a scheduler see the same
// number of earlier blocks between them.
template <int P, int N>
__global__ void __launch_bounds__(SEG_OUT_THREADS, 1)
    ssd_segment_out_kernel(const __nv_bfloat16* __restrict__ xbc, int C, const float* __restrict__ dt_in, int ld_dt, int dt_col0,
                           const float* __restrict__ A_log, const float* __restrict__ dt_bias, const float* __restrict__ Dskip,
                           const float* __restrict__ state, const int32_t* __restrict__ seq_slot, const int32_t* __restrict__ seq_pos0,
                           float* __restrict__ y, int H, int G, const int4* __restrict__ segs, const float* __restrict__ seg_state) {
  griddep_launch();
  griddep_wait();
  constexpr int KS = N / 16, PT = P / 16;  // PT: n8 tiles of a warp's half
  extern __shared__ __align__(16) unsigned char seg_smem[];
  __nv_bfloat16* Cs = reinterpret_cast<__nv_bfloat16*>(seg_smem);  // [128][N + 8]
  __nv_bfloat16* Bs = Cs + SEG_TOKENS * (N + 8);                   // [128][N + 8]
  __nv_bfloat16* Xs = Bs + SEG_TOKENS * (N + 8);                   // [128][P + 8]
  __nv_bfloat16* S3 = Xs + SEG_TOKENS * (P + 8);                   // [3][P][N + 8]: the start state's three terms
  __shared__ float dts[SEG_TOKENS];
  __shared__ float2 cum[SEG_TOKENS];
  __shared__ double part[4];
  const int4 sd = segs[blockIdx.y];
  const int t0 = sd.x, n = sd.y - sd.x, h = blockIdx.x, sq = sd.z;
  if (seg_is_short(sd)) return;
  const int64_t bcol = (int64_t)H * P + (int64_t)(h / (H / G)) * N, ccol = bcol + (int64_t)G * N;
  const float* S_in = (sd.w & SEG_FIRST) ? (seq_pos0[sq] > 0 ? state + ((int64_t)seq_slot[sq] * H + h) * (P * N) : nullptr)
                                         : seg_state + ((int64_t)blockIdx.y * H + h) * (P * N);
  load_rows<N, SEG_OUT_THREADS>(xbc, C, ccol, t0, n, Cs);
  cp_async_commit();
  load_rows<N, SEG_OUT_THREADS>(xbc, C, bcol, t0, n, Bs);
  load_rows<P, SEG_OUT_THREADS>(xbc, C, (int64_t)h * P, t0, n, Xs);
  cp_async_commit();
  if (S_in) {
#pragma unroll 4
    for (int i = threadIdx.x; i < P * N / 4; i += SEG_OUT_THREADS) {
      const float4 v = *reinterpret_cast<const float4*>(S_in + 4 * i);
      uint2 hh, mm, ll;
      split3(make_float2(v.x, v.y), hh.x, mm.x, ll.x);
      split3(make_float2(v.z, v.w), hh.y, mm.y, ll.y);
      __nv_bfloat16* d = S3 + (4 * i / N) * (N + 8) + (4 * i) % N;
      *reinterpret_cast<uint2*>(d) = hh;
      *reinterpret_cast<uint2*>(d + P * (N + 8)) = mm;
      *reinterpret_cast<uint2*>(d + 2 * P * (N + 8)) = ll;
    }
  }
  segment_decays(dt_in, ld_dt, dt_col0 + h, t0, n, -expf(A_log[h]), dt_bias[h], dts, cum, part);
  const float dsk = Dskip[h];
  cp_async_wait<1>();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = warp >> 3, rb = (warp & 7) < 4 ? warp & 7 : 11 - (warp & 7);
  const int ph = half * (P / 2);
  const bool live = rb * 16 < n;
  const int i0 = rb * 16 + (lane >> 2), i1 = i0 + 8;
  uint32_t cf[KS][4];
  float acc[PT][4];
#pragma unroll
  for (int j = 0; j < PT; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;
  if (live) {
#pragma unroll
    for (int k = 0; k < KS; ++k) ldmatrix_x4(cf[k], smem_u32(Cs + (rb * 16 + (lane & 15)) * (N + 8) + k * 16 + (lane >> 4) * 8));
    if (S_in) {
#pragma unroll
      for (int j = 0; j < PT / 2; ++j) {
        float sum[2][4] = {};
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          float t[2][4] = {};
#pragma unroll
          for (int term = 2; term >= 0; --term) {  // smallest first
            uint32_t b[4];
            ldmatrix_x4(b, smem_u32(S3 + (term * P + ph + j * 16 + ((lane >> 4) & 1) * 8 + (lane & 7)) * (N + 8) + k * 16 + ((lane >> 3) & 1) * 8));
            mma_bf16_16816(t[0], cf[k], b[0], b[1]);
            mma_bf16_16816(t[1], cf[k], b[2], b[3]);
          }
          add_to(sum[0], t[0]);
          add_to(sum[1], t[1]);
        }
        add_to(acc[2 * j], sum[0]);
        add_to(acc[2 * j + 1], sum[1]);
      }
      const float e0 = expf(cum[i0].x), e1 = expf(cum[i1].x);
      const float d0 = fmaf(e0, cum[i0].y, e0), d1 = fmaf(e1, cum[i1].y, e1);
#pragma unroll
      for (int j = 0; j < PT; ++j) {
        acc[j][0] *= d0;
        acc[j][1] *= d0;
        acc[j][2] *= d1;
        acc[j][3] *= d1;
      }
    }
  }
  cp_async_wait<0>();
  int odd = n > SEG_TOKENS;  // or an infinite or NaN x among those that this thread copied
  for (int i = threadIdx.x; i < SEG_TOKENS * P / 8; i += SEG_OUT_THREADS) {
    const uint4 v = *reinterpret_cast<const uint4*>(Xs + i / (P / 8) * (P + 8) + i % (P / 8) * 8);
    odd |= nonfinite_bf16x2(v.x) | nonfinite_bf16x2(v.y) | nonfinite_bf16x2(v.z) | nonfinite_bf16x2(v.w);
  }
  if (__syncthreads_or(odd)) {
    walk_segment<P, N, true>(xbc, C, dt_in, ld_dt, dt_col0 + h, t0, n, (int64_t)h * P, bcol, ccol, -expf(A_log[h]), dt_bias[h], dsk, S_in,
                             nullptr, y, H * P, nullptr);
    return;
  }
  if (!live) return;
  const float2 ci0 = cum[i0], ci1 = cum[i1];
  for (int jb = 0; jb <= rb; ++jb) {
    float g[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int c = 0; c < 4; ++c) g[u][c] = 0.f;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      uint32_t b[4];
      ldmatrix_x4(b, smem_u32(Bs + (jb * 16 + ((lane >> 4) & 1) * 8 + (lane & 7)) * (N + 8) + k * 16 + ((lane >> 3) & 1) * 8));
      float t[2][4] = {};
      mma_bf16_16816(t[0], cf[k], b[0], b[1]);
      mma_bf16_16816(t[1], cf[k], b[2], b[3]);
      add_to(g[0], t[0]);
      add_to(g[1], t[1]);
    }
    uint32_t ah[4], am[4], al[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j0 = jb * 16 + u * 8 + 2 * (lane & 3);
      const float2 c0 = cum[j0], c1 = cum[j0 + 1];
      const float dt0 = dts[j0], dt1 = dts[j0 + 1];
      float2 m0, m1;
      m0.x = j0 <= i0 ? g[u][0] * (expf((ci0.x - c0.x) + (ci0.y - c0.y)) * dt0) : 0.f;
      m0.y = j0 + 1 <= i0 ? g[u][1] * (expf((ci0.x - c1.x) + (ci0.y - c1.y)) * dt1) : 0.f;
      m1.x = j0 <= i1 ? g[u][2] * (expf((ci1.x - c0.x) + (ci1.y - c0.y)) * dt0) : 0.f;
      m1.y = j0 + 1 <= i1 ? g[u][3] * (expf((ci1.x - c1.x) + (ci1.y - c1.y)) * dt1) : 0.f;
      split3(m0, ah[2 * u], am[2 * u], al[2 * u]);
      split3(m1, ah[2 * u + 1], am[2 * u + 1], al[2 * u + 1]);
    }
#pragma unroll
    for (int j = 0; j < PT / 2; ++j) {
      uint32_t b[4];
      ldmatrix_x4_trans(b, smem_u32(Xs + (jb * 16 + (lane & 15)) * (P + 8) + ph + j * 16 + (lane >> 4) * 8));
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float t[4] = {};
        mma_bf16_16816(t, al, b[2 * u], b[2 * u + 1]);
        mma_bf16_16816(t, am, b[2 * u], b[2 * u + 1]);
        mma_bf16_16816(t, ah, b[2 * u], b[2 * u + 1]);
        add_to(acc[2 * j + u], t);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int i = r ? i1 : i0;
    if (i >= n) continue;
    float* dst = y + (int64_t)(t0 + i) * H * P + (int64_t)h * P + ph + 2 * (lane & 3);
    const __nv_bfloat16* xr = Xs + i * (P + 8) + ph + 2 * (lane & 3);
#pragma unroll
    for (int j = 0; j < PT; ++j) {
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(xr + j * 8));
      *reinterpret_cast<float2*>(dst + j * 8) = make_float2(acc[j][2 * r] + dsk * x.x, acc[j][2 * r + 1] + dsk * x.y);
    }
  }
}

// the slot's new state of every sequence that ran as segments: its last segment's start state, decayed, plus that segment's own.  Runs
// once all segments have read their start states (the first one's is the slot itself).
__global__ void ssd_segment_final_kernel(float* __restrict__ state, const float* __restrict__ seg_state, const float* __restrict__ seg_dtsum,
                                         const float* __restrict__ A_log, const int4* __restrict__ segs, const int32_t* __restrict__ seq_seg0,
                                         const int32_t* __restrict__ seq_slot, const int32_t* __restrict__ seq_pos0, int H, int head_elems) {
  griddep_launch();
  griddep_wait();
  const int sq = blockIdx.y, last = seq_seg0[sq + 1] - 1;
  if (last < seq_seg0[sq] || seg_is_short(segs[last])) return;
  const int64_t per_seq = (int64_t)H * head_elems;
  const int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (e >= per_seq) return;
  const int h = (int)(e / head_elems);
  float4* slot = reinterpret_cast<float4*>(state + (int64_t)seq_slot[sq] * per_seq + e);
  const float d = expf(-expf(A_log[h]) * seg_dtsum[(int64_t)last * H + h]);
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (last > seq_seg0[sq]) s = *reinterpret_cast<const float4*>(seg_state + (int64_t)last * per_seq + e);
  else if (seq_pos0[sq] > 0) s = *slot;
  const float4 l = *reinterpret_cast<const float4*>(seg_state + (int64_t)seq_seg0[sq] * per_seq + e);
  *slot = make_float4(d * s.x + l.x, d * s.y + l.y, d * s.z + l.z, d * s.w + l.w);
}

namespace {

template <int P, int N>
int launch_state(const __nv_bfloat16* xbc, int C, const float* dt_in, int ld_dt, int dt_col0, const float* A_log, const float* dt_bias, int H,
                 int G, const int4* segs, int num_segs, const int32_t* seq_seg0, float* seg_state, float* seg_dtsum, cudaStream_t st) {
  constexpr size_t smem = (size_t)SEG_TOKENS * (P + 8 + N + 8) * 2;
  B200_CUDA_OK(cudaFuncSetAttribute(ssd_segment_state_kernel<P, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  B200_CUDA_OK(launch_kernel(ssd_segment_state_kernel<P, N>, dim3(H, num_segs), dim3(SEG_THREADS), smem, st, xbc, C, dt_in, ld_dt, dt_col0,
                             A_log, dt_bias, H, G, segs, seq_seg0, seg_state, seg_dtsum));
  return B200_OK;
}

template <int P, int N>
int launch_out(const __nv_bfloat16* xbc, int C, const float* dt_in, int ld_dt, int dt_col0, const float* A_log, const float* dt_bias,
               const float* D, const float* state, const int32_t* seq_slot, const int32_t* seq_pos0, float* y, int H, int G, const int4* segs,
               int num_segs, const float* seg_state, cudaStream_t st) {
  constexpr size_t smem = ((size_t)SEG_TOKENS * (2 * (N + 8) + P + 8) + (size_t)3 * P * (N + 8)) * 2;
  B200_CUDA_OK(cudaFuncSetAttribute(ssd_segment_out_kernel<P, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  B200_CUDA_OK(launch_kernel(ssd_segment_out_kernel<P, N>, dim3(H, num_segs), dim3(SEG_OUT_THREADS), smem, st, xbc, C, dt_in, ld_dt, dt_col0,
                             A_log, dt_bias, D, state, seq_slot, seq_pos0, y, H, G, segs, seg_state));
  return B200_OK;
}

}  // namespace

bool ssd_segments_ok(const void* xbc, int x_dtype, int C, const float* state, int P, int N, const float* seg_state, const float* y) {
  return x_dtype == B200_BF16 && (P == 64 || P == 128) && (N == 64 || N == 128) && C % 8 == 0 && !((uintptr_t)xbc & 15) &&
         !((uintptr_t)state & 15) && !((uintptr_t)seg_state & 15) && !((uintptr_t)y & 7);
}

#define SEG_SIZES(CALL)                                  \
  if (P == 128 && N == 128) return CALL(128, 128);       \
  if (P == 128) return CALL(128, 64);                    \
  if (N == 128) return CALL(64, 128);                    \
  return CALL(64, 64)

int ssd_segment_states(const void* xbc, int C, const float* dt_in, int ld_dt, int dt_col0, const float* A_log, const float* dt_bias, int H,
                       int P, int N, int G, const int32_t* segs, int num_segs, const int32_t* seq_seg0, float* seg_state, float* seg_dtsum,
                       cudaStream_t st) {
#define CALL(P_, N_)                                                                                                                  \
  launch_state<P_, N_>((const __nv_bfloat16*)xbc, C, dt_in, ld_dt, dt_col0, A_log, dt_bias, H, G, reinterpret_cast<const int4*>(segs), \
                       num_segs, seq_seg0, seg_state, seg_dtsum, st)
  SEG_SIZES(CALL);
#undef CALL
}

int ssd_segment_outputs(const void* xbc, int C, const float* dt_in, int ld_dt, int dt_col0, const float* A_log, const float* dt_bias,
                        const float* D, float* state, const int32_t* seq_slot, const int32_t* seq_pos0, float* y, int B, int H, int P, int N,
                        int G, const int32_t* segs, int num_segs, const int32_t* seq_seg0, const float* seg_state, const float* seg_dtsum,
                        cudaStream_t st) {
  const int4* sd = reinterpret_cast<const int4*>(segs);
  auto outputs = [&]() -> int {
#define CALL(P_, N_)                                                                                                                      \
  launch_out<P_, N_>((const __nv_bfloat16*)xbc, C, dt_in, ld_dt, dt_col0, A_log, dt_bias, D, state, seq_slot, seq_pos0, y, H, G, sd,       \
                     num_segs, seg_state, st)
    SEG_SIZES(CALL);
#undef CALL
  };
  if (int rc = outputs()) return rc;
  const int64_t quads = (int64_t)H * P * N / 4;
  B200_CUDA_OK(launch_kernel(ssd_segment_final_kernel, dim3((unsigned)((quads + 255) / 256), B), dim3(256), 0, st, state, seg_state, seg_dtsum,
                             A_log, sd, seq_seg0, seq_slot, seq_pos0, H, P * N));
  return B200_OK;
}

}  // namespace b200
