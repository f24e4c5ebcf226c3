// The weight GEMM for a few tokens: out[M, N] = epilogue(a[M, K] . w[N, K]^T), all operand kinds.
//
// At a few tokens a GEMM is its weights' bytes and a chain of latencies, and the decode schedule (gemm_tcgen05.cu) pays the chain: barrier set-up,
// TMA round trips, tensor-memory allocation, partial tiles through a cluster.  Here a weight byte goes from memory into the register that
// mma.sync reads it from: a lane loads 16 contiguous bytes of its row (four lanes a 64-byte piece, two loads a 128-byte line) and takes them
// as the k slots of its fragments -- a sum does not care which k a slot holds, as long as the tokens' fragments are loaded alike.  No
// shared memory before the sums meet, no barrier in the loop, and the first PF k-blocks of every warp are in flight BEFORE
// griddepcontrol.wait: with 16 warps an SM the chip holds 19 MB of the next GEMM's weights while the kernel ahead finishes.
//   * a CTA takes 16 MT weight rows (MT = 2: gate and up rows of a group, or the two halves of a head, which the epilogue needs together) in
//     2 to 16 warps.  K is cut into 16 slices, every 16th line of 128 bytes each: a chain of tensor-core sums per slice, and the chains meet in
//     shared memory in one tree.  16 warps take a slice each, 8 warps two in turn (s and s + 8), fewer warps such pairs one after the other.
//     So a row's sum does not depend on warps, epilogue or timing: the fused calls give the bits of the linear one followed by what they fuse.
#include "gemm_small.cuh"

#include <limits.h>

namespace b200 {

__device__ __forceinline__ uint4 ldg_stream(const uint8_t* p) {  // weights are read once: they pass L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <int KIND>
__device__ __forceinline__ void mma_small(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (KIND == KIND_F8F6F4)
    asm volatile("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else if constexpr (KIND == KIND_I8)
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// four int8 -> two bf16 pairs, in order (exact: 2^23 + 128 + w as a float, less 2^23 + 128)
__device__ __forceinline__ uint2 widen4(uint32_t w) {
  const uint32_t x = w ^ 0x80808080u;
  const float f0 = __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7440)) - 8388736.f, f1 = __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7441)) - 8388736.f;
  const float f2 = __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7442)) - 8388736.f, f3 = __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7443)) - 8388736.f;
  return make_uint2(__byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632), __byte_perm(__float_as_uint(f2), __float_as_uint(f3), 0x7632));
}

// one 64-byte piece of 16 weight rows (lo: row g, hi: row g + 8) against the tokens' piece
template <int KIND>
__device__ __forceinline__ void mma_piece(uint32_t (&d)[4], const uint4& lo, const uint4& hi, const uint4 (&x)[KIND == KIND_WO8 ? 2 : 1]) {
  if constexpr (KIND == KIND_WO8) {
    const uint32_t l[4] = {lo.x, lo.y, lo.z, lo.w}, h[4] = {hi.x, hi.y, hi.z, hi.w};
    const uint32_t b[8] = {x[0].x, x[0].y, x[0].z, x[0].w, x[1].x, x[1].y, x[1].z, x[1].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint2 a = widen4(l[j]), c = widen4(h[j]);
      mma_small<KIND>(d, a.x, c.x, a.y, c.y, b[2 * j], b[2 * j + 1]);
    }
  } else {
    mma_small<KIND>(d, lo.x, hi.x, lo.y, hi.y, x[0].x, x[0].y);
    mma_small<KIND>(d, lo.z, hi.z, lo.w, hi.w, x[0].z, x[0].w);
  }
}

// NT: eights of tokens; MT: 16-row weight tiles; 16 warps on an SM, in CTAs of WARPS
template <int KIND, int EPI, int NT, int MT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
    gemm_small_kernel(const uint8_t* __restrict__ w, const uint8_t* __restrict__ a, const GemmEpilogue ep, int M, int N, int K) {
  constexpr bool WO = KIND == KIND_WO8;
  constexpr int THREADS = WARPS * 32;
  constexpr int XE = WO ? 2 : 1;                                            // activation bytes per weight byte
  constexpr int REDS = WARPS == 16 ? 16 : 8, STEP = REDS;                   // sums that meet, of one slice or two; lines from one of a sum to its next
  constexpr int SETS = WARPS == 16 ? 1 : 2;                                 // slices that a warp takes in turn
  constexpr int PF = small_ahead(MT * NT, WO), TURNS = PF % SETS ? PF * SETS : PF;  // lines of a warp in flight: what 128 registers hold
  constexpr int ROWS = 16 * MT, TOK = 8 * NT, PITCH = TOK + 1;
  constexpr int SIDES = EPI == EPI_LINEAR ? 1 : 2;                          // sums that an epilogue item takes
  constexpr int ITEM_ROWS = ROWS / SIDES, ITEMS = ITEM_ROWS * TOK, PER = (ITEMS + THREADS - 1) / THREADS;
  __shared__ float red[REDS][ROWS * PITCH];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  // first weight row of tile mt
  int row0[MT];
  if constexpr (EPI == EPI_ROPE) {
    const int per = ep.rope.D / 32, head = blockIdx.x / per, j = blockIdx.x - head * per;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) row0[mt] = head * ep.rope.D + j * 16 + mt * (ep.rope.D >> 1);
  } else {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) row0[mt] = blockIdx.x * ROWS + mt * 16;
  }
  const int wrow = K * (KIND == KIND_F16 ? 2 : 1);  // bytes
  const int nkb = (wrow + 127) >> 7;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 wb[PF][MT][4], xb[PF][2][NT][XE];
  const uint8_t* wp[MT][2];
  bool wok[MT][2];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int r = row0[mt] + g + 8 * hi;
      wok[mt][hi] = r < N;
      wp[mt][hi] = w + (int64_t)(r < N ? r : 0) * wrow + c * 16;
    }
  auto load_w = [&](uint4 (&b)[MT][4], int kb) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int off = kb * 128 + p * 64;
      const bool in = off + c * 16 < wrow;  // rows are whole 16-byte pieces
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int hi = 0; hi < 2; ++hi) b[mt][p * 2 + hi] = in && wok[mt][hi] ? ldg_stream(wp[mt][hi] + off) : zero;
    }
  };
  auto load_x = [&](uint4 (&b)[2][NT][XE], int kb) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int off = kb * 128 + p * 64 + c * 16;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int m = nt * 8 + g;
#pragma unroll
        for (int e = 0; e < XE; ++e)
          b[p][nt][e] = off < wrow && m < M ? *reinterpret_cast<const uint4*>(a + ((int64_t)m * wrow + off) * XE + e * 16) : zero;
      }
    }
  };
  constexpr bool BY_LINE = KIND != KIND_F16;  // the second form of the loop below
  // the line behind kb in a warp's order (nkb or more: none)
  auto after = [&](int kb) {
    const int pair = (kb & 7) + WARPS;
    return WARPS >= 8 || kb + STEP < nkb ? kb + STEP : pair < 8 ? pair : nkb;
  };
#pragma unroll
  for (int s = 0, k = warp; s < PF; ++s)
    if (k < nkb) {
      load_w(wb[s], k);
      k = BY_LINE ? after(k) : k + STEP;
    }
  griddep_wait();  // before everything but the weights: scales and biases may be what the kernel ahead has written
#pragma unroll
  for (int s = 0, k = warp; s < PF; ++s)
    if (k < nkb) {
      load_x(xb[s], k);
      k = BY_LINE ? after(k) : k + STEP;
    }
  // the epilogue's operands of this thread's items, while the products are taken
  float wsc[PER][SIDES], bia[PER][SIDES], asc[PER], res[PER], act[PER];
  long long pos[PER], slot[PER];
  const bool hb = ep.bias != nullptr, hr = EPI == EPI_LINEAR && ep.residual != nullptr;
#pragma unroll
  for (int q = 0; q < PER; ++q)
#pragma unroll
    for (int sd = 0; sd < SIDES; ++sd) {
      const int i = threadIdx.x + q * THREADS, n = (SIDES == 1 ? row0[0] : row0[sd % MT]) + i % ITEM_ROWS;
      wsc[q][sd] = i < ITEMS && n < N && ep.w_scale ? ep.w_scale[n] : 1.f;
      bia[q][sd] = i < ITEMS && n < N && hb ? __bfloat162float(ep.bias[n]) : 0.f;
    }
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = threadIdx.x + q * THREADS, m = i / ITEM_ROWS, n = row0[0] + i % ITEM_ROWS;
    const bool ok = i < ITEMS && m < M;
    asc[q] = ok && ep.a_scale ? ep.a_scale[m] : 1.f;
    res[q] = ok && hr && n < N ? __bfloat162float(ep.residual[(int64_t)m * N + n]) : 0.f;
    if constexpr (EPI == EPI_ROPE) {
      pos[q] = ok ? ep.rope.positions[m] : 0;
      slot[q] = ok ? ep.rope.slot_mapping[m] : -1;
      pos[q] = pos[q] < 0 ? 0 : pos[q] >= ep.rope.max_pos ? ep.rope.max_pos - 1 : pos[q];
    }
  }
  uint32_t acc[SETS][MT][NT][4];
  auto clear = [&]() {
#pragma unroll
    for (int t = 0; t < SETS; ++t)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[t][mt][nt][e] = 0u;
  };
  auto leave = [&](float* to) {  // a slice or a pair (in either order, which a sum does not tell)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t v = acc[0][mt][nt][e], u = SETS == 2 ? acc[SETS - 1][mt][nt][e] : 0u;
          to[(mt * 16 + g + (e >= 2 ? 8 : 0)) * PITCH + nt * 8 + 2 * c + (e & 1)] = KIND == KIND_I8 ? __uint_as_float(v + u) : __uint_as_float(v) + __uint_as_float(u);
        }
  };
  auto multiply = [&](uint32_t (&d)[MT][NT][4], int st) {
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_piece<KIND>(d[mt][nt], wb[st][mt][p * 2], wb[st][mt][p * 2 + 1], xb[st][p][nt]);
  };
  auto fetch = [&](int st, int k) {
    load_w(wb[st], k);
    load_x(xb[st], k);
  };
  clear();
  // Two forms of one order, by what the compiler makes of them.  Chained launches of one token, us, constant offsets / line by line: bf16 4096 x 14336
  // 20.1 / 22.2, 28672 x 4096 gate and up 42.0 / 44.0; fp8 16.2 / 14.1 and 27.4 / 26.3, int8 weights 512 x 512 1.9 / 1.6, 55296 x 5120 73 / 70.
  if constexpr (!BY_LINE) {
    for (int kb = warp; kb < nkb;) {  // a turn's offsets from kb and next are constants
      int next = kb + TURNS * STEP;
      const bool end = WARPS < 8 && next >= nkb;  // of a pair; the next one's first lines are fetched meanwhile
      if (end) next = (kb & 7) + WARPS < 8 ? (kb & 7) + WARPS : nkb;
#pragma unroll
      for (int q = 0; q < TURNS; ++q) {
        const int k = kb + q * STEP, ahead = q < TURNS - PF ? k + PF * STEP : next + (q - TURNS + PF) * STEP;
        if (k < nkb) multiply(acc[q % SETS], q % PF);
        if (ahead < nkb) fetch(q % PF, ahead);
      }
      if (end) {
        leave(red[kb & 7]);
        clear();
      }
      kb = next;
    }
  } else {
    int ahead = warp;
#pragma unroll
    for (int s = 0; s < PF; ++s)
      if (ahead < nkb) ahead = after(ahead);
    for (int cur = warp; cur < nkb;)
#pragma unroll
      for (int q = 0; q < TURNS; ++q)
        if (cur < nkb) {
          multiply(acc[q % SETS], q % PF);
          if (ahead < nkb) {
            fetch(q % PF, ahead);
            ahead = after(ahead);
          }
          if (WARPS < 8 && cur + STEP >= nkb) {  // the pair's last line
            leave(red[cur & 7]);
            clear();
          }
          cur = after(cur);
        }
  }
  if (WARPS >= 8) leave(red[warp]);
  // Not earlier: CTAs of the next kernels that wait for this one hold registers that its own CTAs still need (a step of TinyLlama, one
  // sequence, 1071 us with this at the top, 776 here; Llama 3.1 8B fp8, 6 layers, 520 and 510)
  griddep_launch();
  __syncthreads();
  auto total = [&](int r, int t) {
    if constexpr (KIND == KIND_I8) {
      int v = 0;
#pragma unroll
      for (int k = 0; k < REDS; ++k) v += (k & 7) < nkb ? __float_as_int(red[k][r * PITCH + t]) : 0;  // slices without lines were left by nobody
      return (float)v;
    } else {
      float v[REDS];  // by halves: log2 roundings
#pragma unroll
      for (int k = 0; k < REDS; ++k) v[k] = (k & 7) < nkb ? red[k][r * PITCH + t] : 0.f;
#pragma unroll
      for (int o = REDS / 2; o >= 1; o /= 2)
#pragma unroll
        for (int k = 0; k < o; ++k) v[k] += v[k + o];
      return v[0];
    }
  };
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = threadIdx.x + q * THREADS, m = i / ITEM_ROWS, r = i % ITEM_ROWS;
    const bool ok = i < ITEMS && m < M;
    if constexpr (EPI == EPI_LINEAR) {
      const int n = row0[0] + r;
      if (!ok || n >= N) continue;
      const float y = scaled_value(total(r, m), asc[q], wsc[q][0], hb, bia[q][0], hr, res[q]);
      if (ep.out_f32) reinterpret_cast<float*>(ep.out)[(int64_t)m * N + n] = y;
      else reinterpret_cast<__nv_bfloat16*>(ep.out)[(int64_t)m * N + n] = __float2bfloat16_rn(y);
    } else {
      const int mm = i < ITEMS ? m : 0;
      const float lo = __bfloat162float(__float2bfloat16_rn(scaled_value(total(r, mm), asc[q], wsc[q][0], hb, bia[q][0], false, 0.f)));
      const float hi = __bfloat162float(__float2bfloat16_rn(scaled_value(total(16 + r, mm), asc[q], wsc[q][1], hb, bia[q][1], false, 0.f)));
      if constexpr (EPI == EPI_SILU_QUANT) {
        act[q] = ok ? silu_mul_bf16(lo, hi) : 0.f;
      } else if constexpr (EPI == EPI_SILU_MUL) {  // whole groups of 32 rows: N is a multiple of 32
        const float v = silu_mul_bf16(lo, hi);
        float x = fabsf(v);
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
        if (!ok) continue;
        reinterpret_cast<__nv_bfloat16*>(ep.out)[(int64_t)m * (N >> 1) + blockIdx.x * 16 + r] = __float2bfloat16_rn(v);
        if (r == 0) ep.group_amax[(int64_t)m * (N >> 5) + blockIdx.x] = x;
      } else {
        if (!ok) continue;
        const auto& rp = ep.rope;
        const int half = rp.D >> 1, head = row0[0] / rp.D, d = row0[0] - head * rp.D + r;
        const bool is_q = head < rp.Hq, roped = head < rp.Hq + rp.Hkv;
        float o1 = lo, o2 = hi;
        if (roped) {
          const float cc = rp.cos_t[pos[q] * half + d], ss = rp.sin_t[pos[q] * half + d];
          o1 = __fsub_rn(__fmul_rn(lo, cc), __fmul_rn(hi, ss));
          o2 = __fadd_rn(__fmul_rn(hi, cc), __fmul_rn(lo, ss));
        }
        // the row keeps what the GEMM and the rotation kernel leave there: rotated q, k and v as they are
        __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(ep.out) + (int64_t)m * N + row0[0] + r;
        orow[0] = __float2bfloat16_rn(is_q ? o1 : lo);
        orow[half] = __float2bfloat16_rn(is_q ? o2 : hi);
        if (!is_q && slot[q] >= 0 && slot[q] < rp.num_slots) {
          const long long blk = slot[q] / rp.bs;
          const int off = (int)(slot[q] - blk * rp.bs);
          __nv_bfloat16* dst = (roped ? rp.k_pool : rp.v_pool) + ((blk * rp.Hkv + head - rp.Hq - (roped ? 0 : rp.Hkv)) * rp.bs + off) * rp.D + d;
          dst[0] = __float2bfloat16_rn(o1);
          dst[half] = __float2bfloat16_rn(o2);
        }
      }
    }
  }
  if constexpr (EPI == EPI_SILU_QUANT) {  // the tokens' maxima over the whole grid, as in the decode schedule (gemm_tcgen05.cu) and on its state
    unsigned int* arrived = reinterpret_cast<unsigned int*>(ep.fq_state + 128);
    unsigned int* epoch = arrived + 1;
    const unsigned int e0 = *reinterpret_cast<volatile unsigned int*>(epoch);  // stays until this CTA has arrived
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int m = (threadIdx.x + q * THREADS) / ITEM_ROWS;
      float x = fabsf(act[q]);
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
      if (threadIdx.x % ITEM_ROWS == 0 && m < M) atomicMax(&ep.fq_state[m], ((unsigned long long)(e0 + 1u) << 32) | __float_as_uint(x));
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      if (atomicAdd(arrived, 1u) == gridDim.x - 1) {
        atomicExch(arrived, 0u);
        __threadfence();
        atomicAdd(epoch, 1u);
      } else {
        const long long t0 = clock64();
        unsigned int e;
        do {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(e) : "l"(epoch) : "memory");
          if (clock64() - t0 > 4000000000LL) {  // about 2 s: a grid that is not fully resident must not hang
            printf("b200: silu-quant grid barrier timeout block %d epoch %u\n", blockIdx.x, e0);
            __trap();
          }
        } while (e == e0);
      }
      __threadfence();
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int i = threadIdx.x + q * THREADS, m = i / ITEM_ROWS, r = i % ITEM_ROWS;
      if (m >= M) continue;
      const float amax = __uint_as_float((unsigned int)__ldcg(&ep.fq_state[m])), scale = amax > 0.f ? __fdiv_rn(amax, 448.f) : 1.f;
      if (blockIdx.x == 0 && r == 0) ep.out_scale[m] = scale;
      reinterpret_cast<uint8_t*>(ep.out)[(int64_t)m * (N >> 1) + blockIdx.x * 16 + r] = quant_byte<B200_FP8_E4M3>(act[q], scale);
    }
  }
}

// Which calls the kernel takes: up to 8 tokens all of them, 9 to 16 the weight-only ones.  Chained launches over weights larger than L2, us, decode
// schedule / here, one token: bf16 2048 x 2048 4.7 / 3.3, 2048 x 5632 8.4 / 6.2, 11264 x 2048 gate and up 12.6 / 10.0, 4096 x 14336 25.3 / 19.4, 28672 x 4096
// gate and up 44.7 / 41.2; fp8 4.0 / 2.7, 5.8 / 3.9, 8.1 / 7.0, 14.9 / 12.4, 23.2 / 24.2; weight-only 7.1 / 3.0, 11.5 / 4.7, 12.8 / 10.0, 26.1 / 15.8, 38.8 / 34.3.
// Decode steps at 500 tokens of context, one token: TinyLlama bf16 993 / 620; Llama 3.1 8B, 6 layers, bf16 815 / 689, fp8 549 / 452, 8 tokens weight-only
// 829 / 629; Qwen2.5 32B, 2 layers, 4 tokens, bf16 675 / 583, fp8 402 / 371 -- with all of a layer's GEMMs on one schedule: a decode-schedule GEMM behind one
// of these finds no room for its rings.  So weights that alone are slower here (5120 x 27648 fp8 29.8 / 37.5, int8 weights 46 / 56, at 16 tokens 66; 28672 x
// 4096 fp8 23.2 / 24.2) are left here: with the fp8 28672 x 4096 on the decode schedule the 8B step takes 531.
// 9 to 16 tokens load twice the fragments a weight: 16 tokens, 8B bf16 820 / 898, fp8 572 / 667; weight-only, whose decode schedule
// widens in a pass of its own, 847 / 690, TinyLlama 1243 / 768, Qwen 582 / 578.
bool gemm_small_ok(const void* a, const void* w, int epi, int M, int N, int K, int ab_dtype, int head_dim) {
  const int64_t row = (int64_t)K * (ab_dtype == B200_BF16 ? 2 : 1);
  if (M > (ab_dtype == B200_INT8_WO ? 16 : 8) || row % 16 || (((uintptr_t)a | (uintptr_t)w) & 15) || row * 2 > INT_MAX) return false;
  return epi == EPI_LINEAR || epi == EPI_SILU_MUL || (epi == EPI_ROPE && head_dim % 32 == 0);
}

template <int KIND, int EPI, int NT, int MT, int WARPS>
static int launch_small(const void* a, const void* w, const GemmEpilogue& ep, int M, int N, int K, cudaStream_t s) {
  B200_CUDA_OK(launch_kernel(gemm_small_kernel<KIND, EPI, NT, MT, WARPS>, dim3((N + 16 * MT - 1) / (16 * MT)), dim3(WARPS * 32), 0, s,
                             (const uint8_t*)w, (const uint8_t*)a, ep, M, N, K));
  return B200_OK;
}
// CTAs of 16 rows while there is an SM for each (16 warps of it share a long row, or 8), then of 32 rows -- gate and up rows and the halves of a head
// come in 32 -- with as many warps as let all CTAs be resident; where they are many, four each, so that more of them are in flight and the last
// wave is short.  Measured, bf16, one token, us: 2048 x 5632 with 16 / 8 warps 5.1 / 6.2, 2048 x 2048 2.6 / 2.5; 4096 x 14336 32 rows in 16 warps / 16
// rows in 8 19.4 / 20.3, fp8 12.4 / 14.1, 16 tokens on int8 weights 19.9 / 25.0; 6144 x 4096 16 / 32 rows 11.3 / 10.2; 10272 x 2048 8 / 4 warps 10.2 / 9.2, 32000 x
// 2048 22.8 / 21.8.  4 tokens, 4 / 8 / 16 warps, 7168 x 4096 gate
// and up 14.8 / 12.0 / 12.9 (decode schedule 14.3), 11264 x 2048 10.4 / 12.6 / 12.3; heads of 128, 768 x 4096 12.5 / 7.2 / 5.4 (6.8), 6144 x 4096 14.8 / 11.4 / 12.9.
SmallShape gemm_small_shape(int epi, int M, int N, int K, int ab_dtype) {
  const int tiles = (N + 15) / 16, sms = sm_count(), nt = M <= 8 ? 1 : 2;
  const int64_t row = (int64_t)K * (ab_dtype == B200_BF16 ? 2 : 1);
  SmallShape c{2, tiles <= 2 * sms ? 16 : tiles <= 4 * sms ? 8 : 4, 0};
  if (epi == EPI_LINEAR && tiles <= sms) c = {1, row > 4096 ? 16 : 8, 0};
  c.lines = small_ahead(c.tiles * nt, ab_dtype == B200_INT8_WO);
  return c;
}

template <int KIND, int NT>
static int pick_small(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, int ab_dtype, cudaStream_t s) {
  const SmallShape c = gemm_small_shape(epi, M, N, K, ab_dtype);
#define SMALL_GO(EPI, TILES, WARPS) \
  if (epi == EPI && c.tiles == TILES && c.warps == WARPS) return launch_small<KIND, EPI, NT, TILES, WARPS>(a, w, ep, M, N, K, s)
  SMALL_GO(EPI_LINEAR, 1, 16);
  SMALL_GO(EPI_LINEAR, 1, 8);
  SMALL_GO(EPI_LINEAR, 2, 16);
  SMALL_GO(EPI_LINEAR, 2, 8);
  SMALL_GO(EPI_LINEAR, 2, 4);
  SMALL_GO(EPI_SILU_MUL, 2, 16);
  SMALL_GO(EPI_SILU_MUL, 2, 8);
  SMALL_GO(EPI_SILU_MUL, 2, 4);
  SMALL_GO(EPI_ROPE, 2, 16);
  SMALL_GO(EPI_ROPE, 2, 8);
  SMALL_GO(EPI_ROPE, 2, 4);
#undef SMALL_GO
  return B200_ERR_UNSUPPORTED;
}

int launch_gemm_small(const void* a, const void* w, const GemmEpilogue& ep, int epi, int M, int N, int K, int ab_dtype, cudaStream_t s) {
  if (ab_dtype == B200_BF16) return pick_small<KIND_F16, 1>(a, w, ep, epi, M, N, K, ab_dtype, s);
  if (ab_dtype == B200_FP8_E4M3) return pick_small<KIND_F8F6F4, 1>(a, w, ep, epi, M, N, K, ab_dtype, s);
  if (ab_dtype == B200_INT8) return pick_small<KIND_I8, 1>(a, w, ep, epi, M, N, K, ab_dtype, s);
  return M <= 8 ? pick_small<KIND_WO8, 1>(a, w, ep, epi, M, N, K, ab_dtype, s) : pick_small<KIND_WO8, 2>(a, w, ep, epi, M, N, K, ab_dtype, s);
}

// CTAs of two warps: eight an SM, which holds as many weight rows at once as the decode schedule's tiles, and no other CTA meets the barrier
bool small_silu_quant_fits(int N) {
  static const int ctas = [] {
    auto kern = gemm_small_kernel<KIND_F8F6F4, EPI_SILU_QUANT, 1, 2, 2>;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, 64, 0) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    return n * sm_count();
  }();
  return N % 32 == 0 && N / 32 <= ctas;
}
int launch_gemm_small_silu_quant(const void* a, const void* w, const GemmEpilogue& ep, int M, int N, int K, cudaStream_t s) {
  return launch_small<KIND_F8F6F4, EPI_SILU_QUANT, 1, 2, 2>(a, w, ep, M, N, K, s);
}

}  // namespace b200
