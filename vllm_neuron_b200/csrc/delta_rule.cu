// Gated delta-rule recurrence over a ragged batch, beside the selective state-space scan (ssm_scan.cu).
// Per head, token by token, with a matrix state S [D keys x P values] in fp32:
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (o sees the token's own write)
//   * delta_prep: per token, q and k (after their short convolution) become unit vectors per key head,
//     x / sqrt(sum x^2 + unit_eps), q also times q_scale; beta = sigmoid(raw_b), g = exp(-exp(A_log) softplus(raw_a + dt_bias));
//     k . q per key head is kept for the read-out.  Everything fp32.
//   * delta_scan: the columns of S evolve independently (column j only needs v_j), so a CTA owns PC columns of one head of
//     one sequence and L lanes share a column, each keeping R rows in registers: groups of four consecutive rows dealt
//     round-robin to the lanes (lane l holds rows 4 L i + 4 l .. + 3, i < R / 4), so that the lanes of a column read
//     consecutive 16-byte pieces of the staged k and q rows (no bank conflicts) and of the state.  With s_k = S^T k and
//     s_q = S^T q taken BEFORE the update (one pass over the registers, one shuffle tree for both),
//         u = beta (v - g s_k),   S <- g S + k u,   o = g s_q + u (k . q)
//     is the recurrence above, term for term; the kernel takes the tokens two at a time (see the loop), which halves
//     the number of dependent reductions.  Tokens are staged through shared memory in chunks, a ring of DS_STAGES
//     buffers whose cp.async copies run three chunks ahead of the steps (a chunk's steps take about as long as one trip to
//     HBM, so one chunk of lead does not hide it).  State layout [slots][H][P][D] (a column's rows are
//     contiguous), read when the sequence continues (pos0 > 0), zero otherwise, written back at the end of the portion.
#include <math.h>

#include "hybrid_common.cuh"

namespace b200 {

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// one CTA per token: warps take the key heads (unit norms, k . q), threads the value heads (beta, decay)
__global__ void delta_prep_kernel(float* __restrict__ qkv, int ldc, const float* __restrict__ proj, int ldp, int b_col0, int a_col0,
                                  const float* __restrict__ A_log, const float* __restrict__ dt_bias, float* __restrict__ bg,
                                  float* __restrict__ kq, int H, int G, int D, float q_scale, float unit_eps) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int g = warp; g < G; g += nw) {
    float* q = qkv + (int64_t)t * ldc + (int64_t)g * D;
    float* k = q + (int64_t)G * D;
    float sq = 0.f, sk = 0.f;
    for (int i = lane; i < D; i += 32) {
      sq += q[i] * q[i];
      sk += k[i] * k[i];
    }
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    const float iq = q_scale / sqrtf(sq + unit_eps), ik = 1.0f / sqrtf(sk + unit_eps);
    float dot = 0.f;
    for (int i = lane; i < D; i += 32) {
      const float a = q[i] * iq, b = k[i] * ik;
      q[i] = a;
      k[i] = b;
      dot += a * b;
    }
    dot = warp_sum(dot);
    if (lane == 0) kq[(int64_t)t * G + g] = dot;
  }
  for (int h = threadIdx.x; h < H; h += blockDim.x) {
    const float rb = proj[(int64_t)t * ldp + b_col0 + h], ra = proj[(int64_t)t * ldp + a_col0 + h];
    bg[(int64_t)t * 2 * H + h] = 1.0f / (1.0f + expf(-rb));
    bg[(int64_t)t * 2 * H + H + h] = expf(-expf(A_log[h]) * softplus_f(ra + dt_bias[h]));
  }
}

constexpr int DS_THREADS = 128;
constexpr int DS_STAGES = 4;
constexpr int DS_CHUNK = 16;  // tokens staged per shared-memory buffer (fewer when the key rows are long: the two stages must fit)

template <int N>
__device__ __forceinline__ void cp_async_f32(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(src), "n"(N * 4) : "memory");
}

// grid (P / PC column chunks, H, sequences); thread = (column cl = tid / L, lane part l = tid % L), rows 4 L i + 4 l + {0..3}
template <int R>
__global__ void __launch_bounds__(DS_THREADS)
    delta_scan_kernel(const float* __restrict__ qkv, int ldc, const float* __restrict__ bg, const float* __restrict__ kq,
                      float* __restrict__ state, const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_slot,
                      const int32_t* __restrict__ seq_pos0, float* __restrict__ out, int H, int G, int D, int P, int L, int vec4, int CH) {
  griddep_wait();
  const int sq = blockIdx.z, h = blockIdx.y, PC = DS_THREADS / L, c0 = blockIdx.x * PC;
  const int t0 = seq_start[sq], n = seq_start[sq + 1] - t0;
  if (n <= 0) return;
  const int g = h / (H / G);
  const int Dp = L * R;  // padded key length: rows past D stay zero
  extern __shared__ __align__(16) float ds_sm[];
  // per stage: q [CH][Dp] | k [CH][Dp] | v [CH][PC] | beta, decay, k.q [3][CH]
  const int stage_f = CH * (2 * Dp + PC + 3);
  float* o_s = ds_sm + DS_STAGES * stage_f;  // [CH][PC]
  const int tid = threadIdx.x, cl = tid / L, l = tid - cl * L;
  const int col = c0 + cl;
  const bool col_ok = col < P;
  for (int i = tid; i < DS_STAGES * stage_f; i += DS_THREADS) ds_sm[i] = 0.f;  // the pads (rows past D, columns past P) stay zero
  __syncthreads();
  const uint32_t sm0 = smem_u32(ds_sm);
  const int vcols = P - c0 < PC ? P - c0 : PC;
  // this thread's first copy of a chunk and the step to its next one (rows of dq / vq 16-byte pieces, or D / vcols floats):
  // the divisions happen once, not per chunk
  const int dq = vec4 ? D >> 2 : D, vq = vec4 ? vcols >> 2 : vcols;
  const int q_r0 = tid / dq, q_d0 = tid - q_r0 * dq, q_dr = DS_THREADS / dq, q_dd = DS_THREADS - q_dr * dq;
  const int v_r0 = vq > 0 ? tid / vq : CH, v_d0 = vq > 0 ? tid - v_r0 * vq : 0, v_dr = vq > 0 ? DS_THREADS / vq : 0,
            v_dd = vq > 0 ? DS_THREADS - v_dr * vq : 0;
  const float* src_q0 = qkv + (int64_t)t0 * ldc + (int64_t)g * D;
  const float* src_v0 = qkv + (int64_t)t0 * ldc + 2 * (int64_t)G * D + (int64_t)h * P + c0;
  const int64_t k_off = (int64_t)G * D;
  auto issue = [&](int ck) {
    const int i0 = ck * CH;
    const int cnt = n - i0 < CH ? n - i0 : CH;
    if (cnt > 0) {
      const uint32_t base = sm0 + (uint32_t)((ck % DS_STAGES) * stage_f * 4);
      const float* src_q = src_q0 + (int64_t)i0 * ldc;
      const float* src_v = src_v0 + (int64_t)i0 * ldc;
      for (int r = q_r0, d = q_d0; r < cnt;) {
        if (vec4) {
          cp_async_f32<4>(base + (uint32_t)((r * Dp + 4 * d) * 4), src_q + (int64_t)r * ldc + 4 * d);
          cp_async_f32<4>(base + (uint32_t)(((CH + r) * Dp + 4 * d) * 4), src_q + k_off + (int64_t)r * ldc + 4 * d);
        } else {
          cp_async_f32<1>(base + (uint32_t)((r * Dp + d) * 4), src_q + (int64_t)r * ldc + d);
          cp_async_f32<1>(base + (uint32_t)(((CH + r) * Dp + d) * 4), src_q + k_off + (int64_t)r * ldc + d);
        }
        r += q_dr;
        d += q_dd;
        if (d >= dq) {
          d -= dq;
          ++r;
        }
      }
      for (int r = v_r0, d = v_d0; r < cnt;) {
        if (vec4) cp_async_f32<4>(base + (uint32_t)((2 * CH * Dp + r * PC + 4 * d) * 4), src_v + (int64_t)r * ldc + 4 * d);
        else cp_async_f32<1>(base + (uint32_t)((2 * CH * Dp + r * PC + d) * 4), src_v + (int64_t)r * ldc + d);
        r += v_dr;
        d += v_dd;
        if (d >= vq) {
          d -= vq;
          ++r;
        }
      }
      const uint32_t sc = base + (uint32_t)((CH * (2 * Dp + PC)) * 4);
      for (int i = tid; i < cnt; i += DS_THREADS) {
        cp_async_f32<1>(sc + (uint32_t)(i * 4), bg + (int64_t)(t0 + i0 + i) * 2 * H + h);
        cp_async_f32<1>(sc + (uint32_t)((CH + i) * 4), bg + (int64_t)(t0 + i0 + i) * 2 * H + H + h);
        cp_async_f32<1>(sc + (uint32_t)((2 * CH + i) * 4), kq + (int64_t)(t0 + i0 + i) * G + g);
      }
    }
    cp_async_commit();  // an empty group past the end keeps the wait counts uniform
  };
  // ---- state
  float S[R];
  float* srow = state + (((int64_t)seq_slot[sq] * H + h) * P + (col_ok ? col : 0)) * D + 4 * l;
  const int gstep = 4 * L;  // rows between two of this lane's groups of four
#pragma unroll
  for (int r = 0; r < R; ++r) S[r] = 0.f;
  if (seq_pos0[sq] > 0 && col_ok) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((r >> 2) * gstep + 4 * l + (r & 3) < D) S[r] = srow[(r >> 2) * gstep + (r & 3)];
  }
  const int chunks = (n + CH - 1) / CH;
#pragma unroll
  for (int i = 0; i < DS_STAGES - 1; ++i) issue(i);
  for (int ck = 0; ck < chunks; ++ck) {
    issue(ck + DS_STAGES - 1);  // into the stage chunk ck - 1 used: everyone left it at the barrier that ended that chunk
    cp_async_wait<DS_STAGES - 1>();
    __syncthreads();  // chunk ck of every thread has landed; o_s of chunk ck - 1 has been flushed
    const float* st = ds_sm + (ck % DS_STAGES) * stage_f;
    const float* qs = st + 4 * l;
    const float* ks = st + CH * Dp + 4 * l;
    const float* vs = st + 2 * CH * Dp + cl;
    const float* sc = st + CH * (2 * Dp + PC);
    const int cnt = n - ck * CH < CH ? n - ck * CH : CH;
    int c = 0;
    // ---- two tokens per round: with a = S^T k1, b = S^T k2, cq = S^T q1, d = S^T q2 and the scalars e = k1 . k2,
    // f = k1 . q2 (all six reduced over the lanes in ONE shuffle tree),
    //     u1 = beta1 (v1 - g1 a)                 o1 = g1 cq + u1 (k1 . q1)
    //     u2 = beta2 (v2 - g2 (g1 b + e u1))     o2 = g2 (g1 d + f u1) + u2 (k2 . q2)
    //     S <- g1 g2 S + (g2 u1) k1 + u2 k2
    // which is two steps of the recurrence with half the dependent reductions.
    for (; c + 1 < cnt; c += 2) {
      // packed fp32 pairs: rows (r, r + 1) of the state, k and q go through one fma.rn.f32x2 each
      float2 k1[R / 2], k2[R / 2];
      float2 a2 = make_float2(0.f, 0.f), b2 = a2, c2 = a2, d2 = a2, e2 = a2, f2 = a2;
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const int off = c * Dp + (r >> 2) * gstep;
        const float4 ka = *reinterpret_cast<const float4*>(ks + off);
        const float4 qa = *reinterpret_cast<const float4*>(qs + off);
        const float4 kb = *reinterpret_cast<const float4*>(ks + off + Dp);
        const float4 qb = *reinterpret_cast<const float4*>(qs + off + Dp);
        const float2 s0 = make_float2(S[r], S[r + 1]), s1 = make_float2(S[r + 2], S[r + 3]);
        const float2 ka0 = make_float2(ka.x, ka.y), ka1 = make_float2(ka.z, ka.w);
        const float2 kb0 = make_float2(kb.x, kb.y), kb1 = make_float2(kb.z, kb.w);
        const float2 qb0 = make_float2(qb.x, qb.y), qb1 = make_float2(qb.z, qb.w);
        k1[r >> 1] = ka0, k1[(r >> 1) + 1] = ka1;
        k2[r >> 1] = kb0, k2[(r >> 1) + 1] = kb1;
        a2 = ffma2(s1, ka1, ffma2(s0, ka0, a2));
        b2 = ffma2(s1, kb1, ffma2(s0, kb0, b2));
        c2 = ffma2(s1, make_float2(qa.z, qa.w), ffma2(s0, make_float2(qa.x, qa.y), c2));
        d2 = ffma2(s1, qb1, ffma2(s0, qb0, d2));
        e2 = ffma2(ka1, kb1, ffma2(ka0, kb0, e2));
        f2 = ffma2(ka1, qb1, ffma2(ka0, qb0, f2));
      }
      float e0 = e2.x + e2.y, f0 = f2.x + f2.y;
      const float a0 = a2.x, a1 = a2.y, b0 = b2.x, b1 = b2.y, cq0 = c2.x, cq1 = c2.y, d0 = d2.x, d1 = d2.y;
      float a = a0 + a1, b = b0 + b1, cq = cq0 + cq1, d = d0 + d1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        if (o < L) {
          a += __shfl_xor_sync(0xffffffffu, a, o);
          b += __shfl_xor_sync(0xffffffffu, b, o);
          cq += __shfl_xor_sync(0xffffffffu, cq, o);
          d += __shfl_xor_sync(0xffffffffu, d, o);
          e0 += __shfl_xor_sync(0xffffffffu, e0, o);
          f0 += __shfl_xor_sync(0xffffffffu, f0, o);
        }
      }
      const float beta1 = sc[c], g1 = sc[CH + c], kq1 = sc[2 * CH + c];
      const float beta2 = sc[c + 1], g2 = sc[CH + c + 1], kq2 = sc[2 * CH + c + 1];
      const float u1 = beta1 * (vs[c * PC] - g1 * a);
      const float u2 = beta2 * (vs[(c + 1) * PC] - g2 * (g1 * b + e0 * u1));
      const float gg = g1 * g2, w1 = g2 * u1;
      const float2 gg2 = make_float2(gg, gg), w12 = make_float2(w1, w1), u22 = make_float2(u2, u2);
#pragma unroll
      for (int r = 0; r < R; r += 2) {
        const float2 sn = ffma2(k2[r >> 1], u22, ffma2(k1[r >> 1], w12, fmul2(gg2, make_float2(S[r], S[r + 1]))));
        S[r] = sn.x;
        S[r + 1] = sn.y;
      }
      if (l == 0) {
        o_s[c * PC + cl] = g1 * cq + u1 * kq1;
        o_s[(c + 1) * PC + cl] = g2 * (g1 * d + f0 * u1) + u2 * kq2;
      }
    }
    if (c < cnt) {  // an odd token left
      float kr[R];
      float pk0 = 0.f, pk1 = 0.f, pq0 = 0.f, pq1 = 0.f;
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(ks + c * Dp + (r >> 2) * gstep);
        const float4 q4 = *reinterpret_cast<const float4*>(qs + c * Dp + (r >> 2) * gstep);
        kr[r] = k4.x, kr[r + 1] = k4.y, kr[r + 2] = k4.z, kr[r + 3] = k4.w;
        pk0 += S[r] * k4.x + S[r + 2] * k4.z;
        pk1 += S[r + 1] * k4.y + S[r + 3] * k4.w;
        pq0 += S[r] * q4.x + S[r + 2] * q4.z;
        pq1 += S[r + 1] * q4.y + S[r + 3] * q4.w;
      }
      float pk = pk0 + pk1, pq = pq0 + pq1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        if (o < L) {  // L is a power of two, the same for every thread
          pk += __shfl_xor_sync(0xffffffffu, pk, o);
          pq += __shfl_xor_sync(0xffffffffu, pq, o);
        }
      }
      const float beta = sc[c], gd = sc[CH + c], dkq = sc[2 * CH + c];
      const float u = beta * (vs[c * PC] - gd * pk);
#pragma unroll
      for (int r = 0; r < R; ++r) S[r] = gd * S[r] + kr[r] * u;
      if (l == 0) o_s[c * PC + cl] = gd * pq + u * dkq;
    }
    __syncthreads();  // o_s complete; everyone is done with this stage before the next iteration copies a later chunk into it
    for (int i = tid; i < cnt * vcols; i += DS_THREADS) {
      const int r = i / vcols, d = i - r * vcols;
      out[((int64_t)(t0 + ck * CH + r) * H + h) * P + c0 + d] = o_s[r * PC + d];
    }
  }
  // the next kernel of the stream may take SM slots from here on: earlier, its waiting CTAs would displace this kernel's own
  griddep_launch();
  cp_async_wait<0>();
  if (col_ok) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((r >> 2) * gstep + 4 * l + (r & 3) < D) srow[(r >> 2) * gstep + (r & 3)] = S[r];
  }
}

// Prompt portions in ROUNDS OF EIGHT tokens (D = 16 R = 64 or 128 keys, P a multiple of 16).  With S the state before a round,
// a_i = S^T k_i and c_i = S^T q_i come from one pass over the registers, and the recurrence then runs on these numbers alone:
// after token j every later token i of the round has
//     a_i <- g_j a_i + u_j (k_j . k_i),   c_i <- g_j c_i + u_j (k_j . q_i),     u_i = beta_i (v_i - g_i a_i),   o_i = c_i,
// which is S_j^T k_i and S_j^T q_i term for term, and S <- (g_1 .. g_8) S + sum_j (g_{j+1} .. g_8) u_j k_j closes the round.
// The two-token rounds of the kernel above are bound by what every column repeats: two of its six dot products (k1 . k2,
// k1 . q2) are the same for all columns, each value takes a whole shuffle tree, and a staged k or q serves one column.  Here
//   * a lane keeps 2 columns x R rows (16 lanes per column pair, rows 64 i + 4 l + {0..3}), so a shared-memory read serves two
//     columns; the 32 sums of a round are reduced by halving (30 shuffles for 32 sums, not 4 each), which leaves lane
//     8 c + i of the pair with a_i and c_i of column c: the eight lanes of a column then walk the tokens, one shuffle each;
//   * the products k_j . k_i and k_j . q_i are taken once per CTA, one chunk of 16 tokens AHEAD, by four warps of their own
//     (one per round of the chunk and kk / kq) that also issue the copies, so that one barrier per chunk covers the copies,
//     the products and the stages.  These warps fold the decays between the two tokens into the products, which leaves one
//     multiply-add per token and column in the serial walk, and carry the products of decays that scale a, c and S with
//     their rounding errors: so the walk rounds less often than the two-token rounds do.
// Error against 64 bits over those sizes: outputs 0.93 - 0.95 of the two-token kernel's, states 0.85 - 0.94.  What bounds it is
// still the chain of a round (the sums, the halving, eight dependent steps, the update: about 1 us at 128 keys with one CTA on the SM).
// A CTA is 16 columns (H P / 16 CTAs per sequence: 128 at 16 heads of 128) because the walk is serial in the tokens and only
// columns fill the chip.
constexpr int DR_MAIN = 128, DR_AUX = 128, DR_COLS = 16, DR_CHUNK = 16, DR_STAGES = 4, DR_EF = 96;
__host__ __device__ constexpr int dr_stage_floats(int D) { return DR_CHUNK * (2 * D + DR_COLS + 3); }

template <int N>
__device__ __forceinline__ void load_rows(float (&v)[N], const float* p) {
  if constexpr (N == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x, v[1] = t.y;
  }
}

// The sums of N values over the 2 N / F lanes above, by halving: lane l of its group ends with values F l .. F l + F - 1.
template <int N, int F>
__device__ __forceinline__ void reduce_halving(float (&v)[N], int lane) {
#pragma unroll
  for (int n = N / 2; n >= F; n >>= 1) {
    const int o = n / F;
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i < n) {
        const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
}

// grid (P / 16, H, sequences)
template <int R>
__global__ void __launch_bounds__(DR_MAIN + DR_AUX, 2)
    delta_scan_rounds_kernel(const float* __restrict__ qkv, int ldc, const float* __restrict__ bg, const float* __restrict__ kq,
                             float* __restrict__ state, const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_slot,
                             const int32_t* __restrict__ seq_pos0, float* __restrict__ out, int H, int G, int P) {
  constexpr int D = 16 * R, RE = D / 32, STAGE = dr_stage_floats(D);
  griddep_wait();
  const int sq = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * DR_COLS;
  const int t0 = seq_start[sq], n = seq_start[sq + 1] - t0;
  if (n <= 0) return;
  const int g = h / (H / G);
  if (n == 1) {
    // a decoded token beside the prompts moves the state and little else: all threads, 16 lanes a column, nothing staged
    const int c = c0 + threadIdx.x / 16, r0 = threadIdx.x % 16 * 4;
    const float* row = qkv + (int64_t)t0 * ldc;
    float* sp = state + (((int64_t)seq_slot[sq] * H + h) * P + c) * D + r0;
    const bool old = seq_pos0[sq] > 0;
    float S[R], k[R];
    float a = 0.f, cq = 0.f;
#pragma unroll
    for (int r = 0; r < R; r += 4) {
      const float4 s = old ? *reinterpret_cast<const float4*>(sp + 16 * r) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 q4 = *reinterpret_cast<const float4*>(row + (int64_t)g * D + 16 * r + r0);
      const float4 k4 = *reinterpret_cast<const float4*>(row + (int64_t)(G + g) * D + 16 * r + r0);
      S[r] = s.x, S[r + 1] = s.y, S[r + 2] = s.z, S[r + 3] = s.w;
      k[r] = k4.x, k[r + 1] = k4.y, k[r + 2] = k4.z, k[r + 3] = k4.w;
      a += (s.x * k4.x + s.y * k4.y) + (s.z * k4.z + s.w * k4.w);
      cq += (s.x * q4.x + s.y * q4.y) + (s.z * q4.z + s.w * q4.w);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      cq += __shfl_xor_sync(0xffffffffu, cq, o);
    }
    const float gd = bg[(int64_t)t0 * 2 * H + H + h];
    const float u = bg[(int64_t)t0 * 2 * H + h] * (row[2 * (int64_t)G * D + (int64_t)h * P + c] - gd * a);
    if (r0 == 0) out[((int64_t)t0 * H + h) * P + c] = gd * cq + u * kq[(int64_t)t0 * G + g];
#pragma unroll
    for (int r = 0; r < R; r += 4)
      *reinterpret_cast<float4*>(sp + 16 * r) = make_float4(gd * S[r] + k[r] * u, gd * S[r + 1] + k[r + 1] * u, gd * S[r + 2] + k[r + 2] * u,
                                                            gd * S[r + 3] + k[r + 3] * u);
    return;
  }
  // per stage: q [CHUNK][D] | k [CHUNK][D] | v [CHUNK][COLS] | beta, decay, k.q [3][CHUNK]
  extern __shared__ __align__(16) float ds_sm[];
  // [2 chunks][2 rounds]: pairs (j, i), j < i, kk [32] | kq [32] | g_0 .. g_{i-1} high [8], low [8] | g_{i+1} .. g_7 [8] | g_0 .. g_7
  float* ef = ds_sm + DR_STAGES * STAGE;
  const bool main_warp = threadIdx.x < DR_MAIN;
  const int tid = main_warp ? threadIdx.x : threadIdx.x - DR_MAIN, warp = tid >> 5, lane = tid & 31, l = lane & 15, i8 = lane & 7;
  const uint32_t sm0 = smem_u32(ds_sm);
  const float* src_q0 = qkv + (int64_t)t0 * ldc + (int64_t)g * D;
  const float* src_v0 = qkv + (int64_t)t0 * ldc + 2 * (int64_t)G * D + (int64_t)h * P + c0;
  const int64_t k_off = (int64_t)G * D;
  auto issue = [&](int ck) {
    const int i0 = ck * DR_CHUNK;
    const int cnt = n - i0 < DR_CHUNK ? n - i0 : DR_CHUNK;
    if (cnt > 0) {
      float* st = ds_sm + (ck % DR_STAGES) * STAGE;
      const uint32_t base = sm0 + (uint32_t)((ck % DR_STAGES) * STAGE * 4);
      const float* src_q = src_q0 + (int64_t)i0 * ldc;
#pragma unroll
      for (int i = tid; i < DR_CHUNK * D / 4; i += DR_AUX) {
        const int r = i / (D / 4), d = i % (D / 4) * 4;
        if (r < cnt) {
          cp_async_f32<4>(base + (uint32_t)((r * D + d) * 4), src_q + (int64_t)r * ldc + d);
          cp_async_f32<4>(base + (uint32_t)(((DR_CHUNK + r) * D + d) * 4), src_q + k_off + (int64_t)r * ldc + d);
        } else if (r < ((cnt + 7) & ~7)) {  // the rest of the last round: no keys, no weight, no decay
          *reinterpret_cast<float4*>(st + r * D + d) = make_float4(0.f, 0.f, 0.f, 0.f);
          *reinterpret_cast<float4*>(st + (DR_CHUNK + r) * D + d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      if (tid < DR_CHUNK * DR_COLS / 4) {
        const int r = tid / (DR_COLS / 4), d = tid % (DR_COLS / 4) * 4;
        if (r < cnt) cp_async_f32<4>(base + (uint32_t)((2 * DR_CHUNK * D + r * DR_COLS + d) * 4), src_v0 + (int64_t)(i0 + r) * ldc + d);
        else *reinterpret_cast<float4*>(st + 2 * DR_CHUNK * D + r * DR_COLS + d) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (tid < DR_CHUNK) {
        const int i = tid, o = DR_CHUNK * (2 * D + DR_COLS) + i;
        if (i < cnt) {
          const uint32_t sc = base + (uint32_t)(o * 4);
          cp_async_f32<1>(sc, bg + (int64_t)(t0 + i0 + i) * 2 * H + h);
          cp_async_f32<1>(sc + DR_CHUNK * 4, bg + (int64_t)(t0 + i0 + i) * 2 * H + H + h);
          cp_async_f32<1>(sc + 2 * DR_CHUNK * 4, kq + (int64_t)(t0 + i0 + i) * G + g);
        } else {
          st[o] = 0.f, st[o + DR_CHUNK] = 1.f, st[o + 2 * DR_CHUNK] = 0.f;
        }
      }
    }
    cp_async_commit();  // an empty group past the end keeps the wait counts uniform
  };
  // one round of chunk ck: even warps (g_{j+1} .. g_{i-1}) k_j . k_i and the scales of a, odd ones (g_{j+1} .. g_i) k_j . q_i and
  // the weights of u
  int pj = 0, pi = lane;  // the pair that this lane keeps (none from lane 28 on)
  while (pj < 7 && pi >= 7 - pj) pi -= 7 - pj++;
  pi += pj + 1;
  auto products = [&](int ck) {
    const int rnd = warp >> 1, kq_side = warp & 1;
    if (ck * DR_CHUNK + rnd * 8 >= n) return;  // no token (warp-uniform)
    const float* base = ds_sm + (ck % DR_STAGES) * STAGE;
    const float* st = base + rnd * 8 * D + RE * lane;
    const float* rhs = st + (kq_side ? 0 : DR_CHUNK * D);
    float k[7][RE], v[32];
#pragma unroll
    for (int j = 0; j < 7; ++j) load_rows<RE>(k[j], st + (DR_CHUNK + j) * D);
#pragma unroll
    for (int i = 28; i < 32; ++i) v[i] = 0.f;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
      float x[RE];
      load_rows<RE>(x, rhs + i * D);
#pragma unroll
      for (int j = 0; j < i; ++j) {
        float s = k[j][0] * x[0];
#pragma unroll
        for (int r = 1; r < RE; ++r) s = fmaf(k[j][r], x[r], s);
        v[j * 7 - j * (j - 1) / 2 + i - j - 1] = s;
      }
    }
    reduce_halving<32, 1>(v, lane);
    float* e = ef + ((ck & 1) * 2 + rnd) * DR_EF;
    const float* gs = base + DR_CHUNK * (2 * D + DR_COLS + 1) + rnd * 8;
    float between = 1.f, hi = 1.f, lo = 0.f, after = 1.f;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const float gm = gs[m];
      if (m > pj && m < pi + kq_side) between *= gm;
      if (m < lane) {  // hi + lo: the product of decays with its rounding error
        const float p = hi * gm;
        lo = fmaf(lo, gm, fmaf(hi, gm, -p));
        hi = p;
      }
      if (m > lane) after *= gm;
    }
    e[kq_side * 32 + lane] = v[0] * between;
    if (!kq_side && lane < 8) e[64 + lane] = hi, e[72 + lane] = lo;
    if (kq_side && lane < 8) e[80 + lane] = after;
    if (kq_side && lane == 8) e[88] = hi + lo;
  };
  const int chunks = (n + DR_CHUNK - 1) / DR_CHUNK;
  if (!main_warp) {
#pragma unroll
    for (int i = 0; i < DR_STAGES - 1; ++i) issue(i);
    cp_async_wait<DR_STAGES - 2>();
    named_bar_sync(1, DR_AUX);
    products(0);
    for (int ck = 0; ck < chunks; ++ck) {
      cp_async_wait<DR_STAGES - 3>();
      __syncthreads();  // chunk ck + 1 and the products of chunk ck are there; everyone has left chunk ck - 1
      issue(ck + DR_STAGES - 1);
      products(ck + 1);
    }
    griddep_launch();
    cp_async_wait<0>();
    return;
  }
  // ---- state of columns col, col + 1
  const int colp = (warp * 2 + (lane >> 4)) * 2;
  float2 S[2][R / 2];
  float* srow = state + (((int64_t)seq_slot[sq] * H + h) * P + c0 + colp) * D + 4 * l;
  const bool old = seq_pos0[sq] > 0;
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < R / 4; ++r) {
      const float4 s = old ? *reinterpret_cast<const float4*>(srow + c * D + 64 * r) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[c][2 * r] = make_float2(s.x, s.y);
      S[c][2 * r + 1] = make_float2(s.z, s.w);
    }
  float* orow = out + ((int64_t)t0 * H + h) * P + c0 + colp + (l >> 3);
  for (int ck = 0; ck < chunks; ++ck) {
    __syncthreads();  // as above
    const float* st = ds_sm + (ck % DR_STAGES) * STAGE;
    const int cnt = n - ck * DR_CHUNK < DR_CHUNK ? n - ck * DR_CHUNK : DR_CHUNK;
    for (int c8 = 0; c8 < cnt; c8 += 8) {
      const float* qs = st + c8 * D + 4 * l;
      const float* ks = qs + DR_CHUNK * D;
      const float* sc = st + DR_CHUNK * (2 * D + DR_COLS) + c8;
      const float* e = ef + ((ck & 1) * 2 + (c8 >> 3)) * DR_EF;
      float v[32];  // [column][token][k, q]
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        float2 acc[2][2];
#pragma unroll
        for (int r = 0; r < R / 4; ++r) {
          const float4 k4 = *reinterpret_cast<const float4*>(ks + t * D + 64 * r);
          const float4 q4 = *reinterpret_cast<const float4*>(qs + t * D + 64 * r);
          const float2 k0 = make_float2(k4.x, k4.y), k1 = make_float2(k4.z, k4.w), q0 = make_float2(q4.x, q4.y), q1 = make_float2(q4.z, q4.w);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            acc[c][0] = r ? ffma2(S[c][2 * r], k0, acc[c][0]) : fmul2(S[c][0], k0);
            acc[c][1] = r ? ffma2(S[c][2 * r], q0, acc[c][1]) : fmul2(S[c][0], q0);
            acc[c][0] = ffma2(S[c][2 * r + 1], k1, acc[c][0]);
            acc[c][1] = ffma2(S[c][2 * r + 1], q1, acc[c][1]);
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          v[(c * 8 + t) * 2] = acc[c][0].x + acc[c][0].y;
          v[(c * 8 + t) * 2 + 1] = acc[c][1].x + acc[c][1].y;
        }
      }
      reduce_halving<32, 2>(v, lane);
      // lane 8 c + i of a pair: token i of column c
      const bool live = c8 + i8 < cnt;
      const float beta = sc[i8], gi = sc[DR_CHUNK + i8], kqi = sc[2 * DR_CHUNK + i8], hi = e[64 + i8], lo = e[72 + i8];
      const float bv = beta * st[2 * DR_CHUNK * D + (c8 + i8) * DR_COLS + colp + (l >> 3)], nbg = -beta * gi;
      float a = fmaf(hi, v[0], lo * v[0]), cq = gi * fmaf(hi, v[1], lo * v[1]), u = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = j * 7 - j * (j - 1) / 2 - j - 1;
        const float ekk = i8 > j ? e[row + i8] : 0.f, ekq = i8 > j ? e[32 + row + i8] : kqi;
        const float uj = __shfl_sync(0xffffffffu, live ? fmaf(nbg, a, bv) : 0.f, j, 8);
        a = fmaf(uj, ekk, a);
        if (i8 >= j) cq = fmaf(uj, ekq, cq);
        if (i8 == j) u = uj;
      }
      u *= e[80 + i8];
      const float gall = e[88];
      if (live) orow[(int64_t)(ck * DR_CHUNK + c8 + i8) * H * P] = cq;
      const float2 g2 = make_float2(gall, gall);
      float2 dS[2][R / 2];  // summed apart: the state is rounded once per round
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const float w0 = __shfl_sync(0xffffffffu, u, t, 16), w1 = __shfl_sync(0xffffffffu, u, 8 + t, 16);
        const float2 w[2] = {make_float2(w0, w0), make_float2(w1, w1)};
#pragma unroll
        for (int r = 0; r < R / 4; ++r) {
          const float4 k4 = *reinterpret_cast<const float4*>(ks + t * D + 64 * r);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            dS[c][2 * r] = t ? ffma2(make_float2(k4.x, k4.y), w[c], dS[c][2 * r]) : fmul2(make_float2(k4.x, k4.y), w[c]);
            dS[c][2 * r + 1] = t ? ffma2(make_float2(k4.z, k4.w), w[c], dS[c][2 * r + 1]) : fmul2(make_float2(k4.z, k4.w), w[c]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int r = 0; r < R / 2; ++r) S[c][r] = ffma2(g2, S[c][r], dS[c][r]);
    }
  }
  griddep_launch();  // not earlier: the waiting CTAs of the next kernel would displace this kernel's own
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < R / 4; ++r)
      *reinterpret_cast<float4*>(srow + c * D + 64 * r) =
          make_float4(S[c][2 * r].x, S[c][2 * r].y, S[c][2 * r + 1].x, S[c][2 * r + 1].y);
}

// Steps of one token per sequence: nothing is walked, so the state rows [P][D] pass through registers once as 16-byte pieces, D / 4 lanes a row,
// 8 rows a warp, whose 16 sums are reduced together by halving.  Bound by the state's bytes, read and written: 64 sequences, 16 heads of
// 128 x 128 (134 MB, 20 us), with delta_prep in front, L2 flushed, 64.5 us by the kernel above (staged tokens, two barriers), 27.6 by this one;
// 33 sequences 39.8 / 21.5, 4 sequences 17.4 / 13.3; heads of 64 x 64, 64 sequences 33.6 / 17.3.  Errors as before (o 1.0e-7, S 5.8e-8).
constexpr int DSTEP_ROWS = 8, DSTEP_WARPS = 4;
template <int LANES>
__global__ void __launch_bounds__(DSTEP_WARPS * 32)
    delta_step_kernel(const float* __restrict__ qkv, int ldc, const float* __restrict__ bg, const float* __restrict__ kq,
                      float* __restrict__ state, const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_slot,
                      const int32_t* __restrict__ seq_pos0, float* __restrict__ out, int H, int G, int P) {
  constexpr int D = 4 * LANES, PER = 32 / LANES;
  griddep_launch();
  griddep_wait();
  const int sq = blockIdx.z, h = blockIdx.y, t0 = seq_start[sq], t1 = seq_start[sq + 1];
  if (t0 >= t1) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / LANES, l = lane % LANES, gh = h / (H / G);
  const int row0 = (blockIdx.x * DSTEP_WARPS + warp) * DSTEP_ROWS * PER;  // rows row0 + i PER + sub
  if (row0 >= P) return;
  float* sp = state + (((int64_t)seq_slot[sq] * H + h) * P + row0 + sub) * D + l * 4;
  const bool old = seq_pos0[sq] > 0;
  float4 S[DSTEP_ROWS];
#pragma unroll
  for (int i = 0; i < DSTEP_ROWS; ++i)
    S[i] = old && row0 + i * PER + sub < P ? *reinterpret_cast<const float4*>(sp + (int64_t)i * PER * D) : make_float4(0.f, 0.f, 0.f, 0.f);
  for (int t = t0; t < t1; ++t) {  // one turn in a decode step; a longer portion is only slower
    const float* row = qkv + (int64_t)t * ldc;
    const float4 q = *reinterpret_cast<const float4*>(row + (int64_t)gh * D + l * 4), k = *reinterpret_cast<const float4*>(row + (int64_t)(G + gh) * D + l * 4);
    const float beta = bg[(int64_t)t * 2 * H + h], gd = bg[(int64_t)t * 2 * H + H + h], kqd = kq[(int64_t)t * G + gh];
    float v[2 * DSTEP_ROWS];
#pragma unroll
    for (int i = 0; i < DSTEP_ROWS; ++i) {
      v[i] = (S[i].x * k.x + S[i].y * k.y) + (S[i].z * k.z + S[i].w * k.w);
      v[DSTEP_ROWS + i] = (S[i].x * q.x + S[i].y * q.y) + (S[i].z * q.z + S[i].w * q.w);
    }
    int mine = 0, off = LANES / 2;  // mine: the row whose two sums this lane ends up with
#pragma unroll
    for (int m = DSTEP_ROWS / 2; m >= 1; m /= 2, off /= 2) {
      const bool up = l & off;
      mine += up ? m : 0;
#pragma unroll
      for (int i = 0; i < m; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float* b = v + e * DSTEP_ROWS;
          const float keep = up ? b[i + m] : b[i], give = up ? b[i] : b[i + m];
          b[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
    }
#pragma unroll
    for (int o = LANES / 2 / DSTEP_ROWS; o >= 1; o /= 2) {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      v[DSTEP_ROWS] += __shfl_xor_sync(0xffffffffu, v[DSTEP_ROWS], o);
    }
    const int p = row0 + mine * PER + sub;
    const float u = p < P ? beta * (row[2 * (int64_t)G * D + (int64_t)h * P + p] - gd * v[0]) : 0.f;
    if (l % (LANES / DSTEP_ROWS) == 0 && p < P) out[((int64_t)t * H + h) * P + p] = gd * v[DSTEP_ROWS] + u * kqd;
#pragma unroll
    for (int i = 0; i < DSTEP_ROWS; ++i) {
      // row i's value sits in the lanes whose bits spell i
      const float w = __shfl_sync(0xffffffffu, u, sub * LANES + ((i & 4) ? LANES / 2 : 0) + ((i & 2) ? LANES / 4 : 0) + ((i & 1) ? LANES / 8 : 0));
      S[i] = make_float4(fmaf(gd, S[i].x, k.x * w), fmaf(gd, S[i].y, k.y * w), fmaf(gd, S[i].z, k.z * w), fmaf(gd, S[i].w, k.w * w));
    }
  }
#pragma unroll
  for (int i = 0; i < DSTEP_ROWS; ++i)
    if (row0 + i * PER + sub < P) *reinterpret_cast<float4*>(sp + (int64_t)i * PER * D) = S[i];
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_delta_prep(float* qkv, int ldc, const float* proj, int ldp, int b_col0, int a_col0, const float* A_log,
                    const float* dt_bias, float* beta_decay, float* kq, int T, int H, int G, int D, float q_scale, float unit_eps,
                    void* stream) {
  B200_REQUIRE(qkv && proj && A_log && dt_bias && beta_decay && kq, "delta_prep: null pointer");
  B200_REQUIRE(H > 0 && G > 0 && H % G == 0 && D > 0, "delta_prep: %d heads over %d key heads of %d", H, G, D);
  if (T <= 0) return B200_OK;
  B200_CUDA_OK(launch_kernel(delta_prep_kernel, dim3(T), dim3(128), 0, (cudaStream_t)stream, qkv, ldc, proj, ldp, b_col0, a_col0,
                             A_log, dt_bias, beta_decay, kq, H, G, D, q_scale, unit_eps));
  return B200_OK;
}

int b200_delta_scan(const float* qkv, int ldc, const float* beta_decay, const float* kq, float* state, const int32_t* seq_start,
                    const int32_t* seq_slot, const int32_t* seq_pos0, float* out, int B, int max_new, int H, int G, int D, int P,
                    void* stream) {
  B200_REQUIRE(qkv && beta_decay && kq && state && seq_start && seq_slot && seq_pos0 && out, "delta_scan: null pointer");
  B200_REQUIRE(H > 0 && G > 0 && H % G == 0, "delta_scan: %d heads over %d key heads", H, G);
  B200_REQUIRE(D >= 1 && D <= 1024 && P >= 1, "delta_scan: key size %d (1..1024 supported)", D);
  if (B <= 0) return B200_OK;
  // decode steps on rows of whole 16-byte pieces (the kernel's own condition)
  if (max_new == 1 && (D == 64 || D == 128) && ldc % 4 == 0 && H <= 65535 && B <= 65535 && !(((uintptr_t)qkv | (uintptr_t)state) & 15)) {
    const int rows = DSTEP_WARPS * DSTEP_ROWS * (128 / D);
    const dim3 grid((P + rows - 1) / rows, H, B);
#define DSTEP_LAUNCH(LANES)                                                                                                               \
  B200_CUDA_OK(launch_kernel(delta_step_kernel<LANES>, grid, dim3(DSTEP_WARPS * 32), 0, (cudaStream_t)stream, qkv, ldc, beta_decay, kq,   \
                             state, seq_start, seq_slot, seq_pos0, out, H, G, P))
    if (D == 128) DSTEP_LAUNCH(32);
    else DSTEP_LAUNCH(16);
#undef DSTEP_LAUNCH
    return B200_OK;
  }
  // Rounds of eight tokens once a portion fills one; shorter steps stay with the kernel that lets more CTAs share an SM.  Two-token
  // rounds -> rounds of eight at 16 heads of 128 x 128: one portion of 8 tokens 10.2 -> 9.6 us, of 4096 936 -> 522, eight of 512
  // 503 -> 367, 32 of 8 61 -> 59, one of 8 beside 31 decoded tokens 37 -> 31, 1210 and 333 beside 29 decoded tokens 392 -> 246; 8 heads of
  // 64 x 64, 2048 tokens: 451 -> 174.
  if (max_new >= 8 && (D == 64 || D == 128) && P % DR_COLS == 0 && ldc % 4 == 0 && !(((uintptr_t)qkv | (uintptr_t)state) & 15)) {
    const size_t smem = (size_t)(DR_STAGES * dr_stage_floats(D) + 4 * DR_EF) * 4;
    const dim3 grid(P / DR_COLS, H, B);
#define DR_LAUNCH(RR)                                                                                                         \
  do {                                                                                                                       \
    if (smem > 48 * 1024)                                                                                                    \
      B200_CUDA_OK(cudaFuncSetAttribute(delta_scan_rounds_kernel<RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    B200_CUDA_OK(launch_kernel_serial(delta_scan_rounds_kernel<RR>, grid, dim3(DR_MAIN + DR_AUX), smem, (cudaStream_t)stream, qkv, ldc, \
                                      beta_decay, kq, state, seq_start, seq_slot, seq_pos0, out, H, G, P));                  \
  } while (0)
    if (D == 128) DR_LAUNCH(8);
    else DR_LAUNCH(4);
#undef DR_LAUNCH
    return B200_OK;
  }
  // L lanes per column (a power of two), R rows per lane.  More rows per lane mean fewer shuffles and shared-memory reads
  // per multiply-add but fewer warps to hide their latency.  Measured at D = 128, 16 heads: one 4096-token portion 1.38 /
  // 0.97 / 1.27 ms at 32 / 16 / 8 rows per lane; 64 single tokens 0.057 / 0.057 / 0.099 ms (they mostly move the state).
  const int rows_target = max_new > 4 ? 16 : 32;
  int L = 1;
  while (L < 32 && L * rows_target < D) L <<= 1;
  const int need = (D + L - 1) / L;
  const int R = need <= 8 ? 8 : need <= 16 ? 16 : 32;
  const int PC = DS_THREADS / L;
  const int vcols_min = P % PC ? P % PC : PC;
  const int vec4 = D % 4 == 0 && ldc % 4 == 0 && P % 4 == 0 && PC % 4 == 0 && vcols_min % 4 == 0 && !((uintptr_t)qkv & 15);
  int CH = DS_CHUNK;
  while (CH > 4 && (size_t)(DS_STAGES * CH * (2 * L * R + PC + 3) + CH * PC) * 4 > 160 * 1024) CH >>= 1;
  const size_t smem = (size_t)(DS_STAGES * CH * (2 * L * R + PC + 3) + CH * PC) * 4;
  dim3 grid((P + PC - 1) / PC, H, B);
  cudaStream_t st = (cudaStream_t)stream;
#define DS_LAUNCH(RR)                                                                                                        \
  do {                                                                                                                       \
    if (smem > 48 * 1024)                                                                                                    \
      B200_CUDA_OK(cudaFuncSetAttribute(delta_scan_kernel<RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));     \
    B200_CUDA_OK(launch_kernel_serial(delta_scan_kernel<RR>, grid, dim3(DS_THREADS), smem, st, qkv, ldc, beta_decay, kq,    \
                                      state, seq_start, seq_slot, seq_pos0, out, H, G, D, P, L, vec4, CH));                 \
  } while (0)
  if (R == 8) DS_LAUNCH(8);
  else if (R == 16) DS_LAUNCH(16);
  else DS_LAUNCH(32);
#undef DS_LAUNCH
  return B200_OK;
}

}  // extern "C"
