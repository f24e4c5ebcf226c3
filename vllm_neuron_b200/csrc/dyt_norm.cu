// Elementwise and per-row kernels of the hybrid decoder: scaled embedding gather into the fp32 residual stream,
// Dynamic-Tanh norm (gain * tanh(a x) + shift, elementwise, no row statistics), the fused "residual += norm(branch); next = norm(residual)"
// step, the gated grouped RMS norm that closes a state-space mixer, and the clamped gated-linear-unit activation.
// The residual stream and all norm arithmetic are fp32; outputs that feed a GEMM are written in the GEMM operand type.
#include "hybrid_common.cuh"

namespace b200 {

template <typename WT>
__global__ void embed_scale_kernel(const int32_t* __restrict__ tokens, const WT* __restrict__ table, float* __restrict__ out,
                                   int W, int V, float scale) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x;
  int tok = tokens[t];
  tok = tok < 0 ? 0 : (tok >= V ? V - 1 : tok);
  for (int i = threadIdx.x; i < W; i += blockDim.x) out[(int64_t)t * W + i] = ldf(table, (int64_t)tok * W + i) * scale;
}

// four columns at a time (4096 x 2048 from bf16: 19.7 -> 9.9 us)
template <typename WT>
__global__ void embed_scale_vec_kernel(const int32_t* __restrict__ tokens, const WT* __restrict__ table, float* __restrict__ out, int W, int V,
                                       float scale) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x;
  int tok = tokens[t];
  tok = tok < 0 ? 0 : (tok >= V ? V - 1 : tok);
#pragma unroll 2
  for (int i = threadIdx.x * 4; i < W; i += blockDim.x * 4) {
    const float4 v = ldf4(table, (int64_t)tok * W + i);
    *reinterpret_cast<float4*>(out + (int64_t)t * W + i) = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
  }
}

template <typename OT>
__global__ void dyt_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float alpha,
                           OT* __restrict__ out, int W, int64_t total) {
  griddep_launch();
  griddep_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % W);
    stf(out, i, tanhf(alpha * x[i]) * w[c] + b[c]);
  }
}

// the same, four columns a thread, which walks down the rows (4096 x 2048 to bf16: 24.0 -> 9.0 us)
template <typename OT>
__global__ void dyt_vec_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float alpha,
                               OT* __restrict__ out, int W, int T) {
  griddep_launch();
  griddep_wait();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c >= W) return;
  const float4 u = ldf4(w, c), v = ldf4(b, c);
#pragma unroll 2
  for (int t = blockIdx.y; t < T; t += gridDim.y) {
    const float4 r = ldf4(x, (int64_t)t * W + c);
    stf4(out, (int64_t)t * W + c, make_float4(tanhf(alpha * r.x) * u.x + v.x, tanhf(alpha * r.y) * u.y + v.y, tanhf(alpha * r.z) * u.z + v.z,
                                              tanhf(alpha * r.w) * u.w + v.w));
  }
}

// x[t] += dyt1( sum_{c < nsum} y[(t * nsum + c)] + y2[t] );   out2[t] = dyt2(x[t])  (when out2 is given)
template <typename OT>
__global__ void dyt_residual_kernel(float* __restrict__ x, const float* __restrict__ y, int nsum, const float* __restrict__ y2,
                                    const float* __restrict__ w1, const float* __restrict__ b1, float a1,
                                    const float* __restrict__ w2, const float* __restrict__ b2, float a2, OT* __restrict__ out2,
                                    int W, int64_t total) {
  griddep_launch();
  griddep_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / W;
    const int c = (int)(i - t * W);
    float s = 0.f;
    for (int k = 0; k < nsum; ++k) s += y[(t * nsum + k) * W + c];
    if (y2) s += y2[i];
    const float r = x[i] + (tanhf(a1 * s) * w1[c] + b1[c]);
    x[i] = r;
    if (out2) stf(out2, i, tanhf(a2 * r) * w2[c] + b2[c]);
  }
}

// The same four columns at a time: a thread keeps its columns' weights and walks down the rows, so that nothing is divided and every access
// is a vector (4096 x 2048 with expert rows: 57 -> 29 us on average over a layer; one scalar and a 64-bit division per element before).
// NS: nsum where it is known at compile time (0: any), so that two rows' loads go out together (4096 x 2048, one
// row of y: 18.3 us, at its bytes).
template <typename OT, int NS>
__global__ void dyt_residual_vec_kernel(float* __restrict__ x, const float* __restrict__ y, int nsum_, const float* __restrict__ y2,
                                        const float* __restrict__ w1, const float* __restrict__ b1, float a1,
                                        const float* __restrict__ w2, const float* __restrict__ b2, float a2, OT* __restrict__ out2,
                                        int W, int T) {
  const int nsum = NS ? NS : nsum_;
  griddep_launch();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  griddep_wait();  // before the weights too: they may be what the kernel ahead has written
  if (c >= W) return;
  const float4 u1 = ldf4(w1, c), v1 = ldf4(b1, c);
  float4 u2 = make_float4(0.f, 0.f, 0.f, 0.f), v2 = u2;
  if (out2) u2 = ldf4(w2, c), v2 = ldf4(b2, c);
#pragma unroll 2
  for (int t = blockIdx.y; t < T; t += gridDim.y) {
    const int64_t i = (int64_t)t * W + c;
    float4 r = ldf4(x, i), s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < nsum; ++k) {
      const float4 v = ldf4(y, ((int64_t)t * nsum + k) * W + c);
      s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
    }
    if (y2) {
      const float4 v = ldf4(y2, i);
      s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
    }
    r.x += tanhf(a1 * s.x) * u1.x + v1.x;
    r.y += tanhf(a1 * s.y) * u1.y + v1.y;
    r.z += tanhf(a1 * s.z) * u1.z + v1.z;
    r.w += tanhf(a1 * s.w) * u1.w + v1.w;
    *reinterpret_cast<float4*>(x + i) = r;
    if (out2)
      stf4(out2, i, make_float4(tanhf(a2 * r.x) * u2.x + v2.x, tanhf(a2 * r.y) * u2.y + v2.y, tanhf(a2 * r.z) * u2.z + v2.z,
                                tanhf(a2 * r.w) * u2.w + v2.w));
  }
}

// r = y * silu(z) is formed FIRST; then every one of the `ng` equal slices r_k of a row is scaled by
// rsqrt(mean(r_k^2) + eps) and multiplied by w.
template <typename OT>
__global__ void gated_group_rmsnorm_kernel(const float* __restrict__ y, const float* __restrict__ z, int ldz,
                                           const float* __restrict__ w, OT* __restrict__ out, int inner, int ng, float eps) {
  griddep_launch();
  griddep_wait();
  extern __shared__ float sv[];
  __shared__ float red[32];
  const int t = blockIdx.x, g = blockIdx.y, gs = inner / ng;
  const float* yr = y + (int64_t)t * inner + g * gs;
  const float* zr = z + (int64_t)t * ldz + g * gs;
  float ss = 0.f;
  for (int i = threadIdx.x; i < gs; i += blockDim.x) {
    const float v = yr[i] * silu_f(zr[i]);
    sv[i] = v;
    ss += v * v;
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    v = warp_sum(v);
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  const float inv = 1.0f / sqrtf(red[0] / (float)gs + eps);
  for (int i = threadIdx.x; i < gs; i += blockDim.x)
    stf(out, (int64_t)t * inner + g * gs + i, sv[i] * inv * w[g * gs + i]);
}

// The same with a warp per (token, slice), the slice in its registers: 16-byte accesses, no barrier (4096 x 8 slices of 512: 79 -> 37
// us).  Slices of up to 128 V, and enough of them: a warp alone walks a wide slice more slowly than the CTA above does (CTA / warp, us: slices
// of 1024, 4 of them 2.9 / 4.8, 1024 5.3 / 5.7, 1600 6.6 / 6.3; of 512, 64 2.2 / 3.1, 800 3.8 / 3.4; of 256, 64 2.0 / 2.3, 400 2.4 / 2.3).
template <typename OT, int V>
__global__ void gated_group_rmsnorm_warp_kernel(const float* __restrict__ y, const float* __restrict__ z, int ldz,
                                                const float* __restrict__ w, OT* __restrict__ out, int inner, int ng, float eps, int T) {
  griddep_launch();
  griddep_wait();
  const int lane = threadIdx.x & 31, g = blockIdx.y, gs = inner / ng;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  const float* yr = y + (int64_t)t * inner + g * gs;
  const float* zr = z + (int64_t)t * ldz + g * gs;
  float4 v[V];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int i = 4 * (lane + 32 * k);
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < gs) {
      const float4 a = ldf4(yr, i), b = ldf4(zr, i);
      v[k] = make_float4(a.x * silu_f(b.x), a.y * silu_f(b.y), a.z * silu_f(b.z), a.w * silu_f(b.w));
    }
    ss += v[k].x * v[k].x + v[k].y * v[k].y + (v[k].z * v[k].z + v[k].w * v[k].w);
  }
  ss = warp_sum(ss);
  const float inv = 1.0f / sqrtf(ss / (float)gs + eps);
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int i = 4 * (lane + 32 * k);
    if (i >= gs) continue;
    const float4 q = ldf4(w, g * gs + i);
    stf4(out, (int64_t)t * inner + g * gs + i,
         make_float4(v[k].x * inv * q.x, v[k].y * inv * q.y, v[k].z * inv * q.z, v[k].w * inv * q.w));
  }
}

// gu [T, 2 ff] (gate columns first): out = min(g, limit) * sigmoid(1.702 g') * (clamp(u, -limit, limit) + 1), g' the clamped gate
template <typename OT>
__global__ void clamped_glu_kernel(const float* __restrict__ gu, OT* __restrict__ out, int ff, float limit, int64_t total) {
  griddep_launch();
  griddep_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / ff;
    const int c = (int)(i - t * ff);
    const float g = fminf(gu[t * 2 * ff + c], limit);
    const float u = fminf(fmaxf(gu[t * 2 * ff + ff + c], -limit), limit);
    stf(out, i, g / (1.0f + expf(-1.702f * g)) * (u + 1.0f));
  }
}

template <typename OT>
__global__ void clamped_glu_vec_kernel(const float* __restrict__ gu, OT* __restrict__ out, int ff, float limit, int T) {
  griddep_launch();
  griddep_wait();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c >= ff) return;
#pragma unroll 2
  for (int t = blockIdx.y; t < T; t += gridDim.y) {
    const float4 g4 = ldf4(gu, (int64_t)t * 2 * ff + c), u4 = ldf4(gu, (int64_t)t * 2 * ff + ff + c);
    auto one = [&](float g, float u) {
      g = fminf(g, limit);
      u = fminf(fmaxf(u, -limit), limit);
      return g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
    };
    stf4(out, (int64_t)t * ff + c, make_float4(one(g4.x, u4.x), one(g4.y, u4.y), one(g4.z, u4.z), one(g4.w, u4.w)));
  }
}

// rows of `quads` vectors: CTAs of up to 256 threads across a row, and enough rows in flight for two full waves of them
static inline dim3 vec_grid(int quads, int threads, int T) {
  const int x = (quads + threads - 1) / threads;
  const int rows = 148 * 2 * (2048 / threads) / x;
  return dim3(x, T < rows ? T : rows < 1 ? 1 : rows);
}
static inline int vec_threads(int quads) { return quads >= 256 ? 256 : (quads + 31) / 32 * 32; }

static inline int flat_grid(int64_t total, int threads) {
  int64_t b = (total + threads - 1) / threads;
  return (int)(b > 148 * 16 ? 148 * 16 : (b < 1 ? 1 : b));
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_embed_scale(const int32_t* tokens, const void* table, int table_dtype, float* out, int T, int W, int V, float scale,
                     void* stream) {
  B200_REQUIRE(tokens && table && out, "embed_scale: null pointer");
  if (T <= 0) return B200_OK;
  if (W % 4 == 0 && vec4_ok(table, table_dtype == B200_BF16 ? 2 : 4) && vec4_ok(out)) {
    B200_DISPATCH_ELEM(table_dtype, WT,
                       B200_CUDA_OK(launch_kernel(embed_scale_vec_kernel<WT>, dim3(T), dim3(vec_threads(W / 4)), 0, (cudaStream_t)stream, tokens,
                                                  (const WT*)table, out, W, V, scale)));
    return B200_OK;
  }
  B200_DISPATCH_ELEM(table_dtype, WT,
                     B200_CUDA_OK(launch_kernel(embed_scale_kernel<WT>, dim3(T), dim3(256), 0, (cudaStream_t)stream, tokens,
                                                (const WT*)table, out, W, V, scale)));
  return B200_OK;
}

int b200_dyt_norm(const float* x, const float* w, const float* b, float alpha, void* out, int out_dtype, int T, int W,
                  void* stream) {
  B200_REQUIRE(x && w && b && out, "dyt_norm: null pointer");
  if (T <= 0) return B200_OK;
  const int64_t total = (int64_t)T * W;
  if (W % 4 == 0 && vec4_ok(x) && vec4_ok(w) && vec4_ok(b) && vec4_ok(out, out_dtype == B200_BF16 ? 2 : 4)) {
    const int th = vec_threads(W / 4);
    B200_DISPATCH_ELEM(out_dtype, OT,
                       B200_CUDA_OK(launch_kernel(dyt_vec_kernel<OT>, vec_grid(W / 4, th, T), dim3(th), 0, (cudaStream_t)stream, x, w, b, alpha,
                                                  (OT*)out, W, T)));
    return B200_OK;
  }
  B200_DISPATCH_ELEM(out_dtype, OT,
                     B200_CUDA_OK(launch_kernel(dyt_kernel<OT>, dim3(flat_grid(total, 256)), dim3(256), 0, (cudaStream_t)stream,
                                                x, w, b, alpha, (OT*)out, W, total)));
  return B200_OK;
}

int b200_dyt_residual(float* x, const float* y, int nsum, const float* y2, const float* w1, const float* b1, float alpha1,
                      const float* w2, const float* b2, float alpha2, void* out2, int out_dtype, int T, int W, void* stream) {
  B200_REQUIRE(x && y && w1 && b1 && nsum >= 1, "dyt_residual: null pointer");
  B200_REQUIRE(!out2 || (w2 && b2), "dyt_residual: the second norm needs its weight and bias");
  if (T <= 0) return B200_OK;
  const int64_t total = (int64_t)T * W;
  const int oes = out_dtype == B200_BF16 ? 2 : 4;
  if (W % 4 == 0 && vec4_ok(x) && vec4_ok(y) && vec4_ok(y2) && vec4_ok(w1) && vec4_ok(b1) && vec4_ok(w2) && vec4_ok(b2) && vec4_ok(out2, oes)) {
    const int th = vec_threads(W / 4);
    B200_DISPATCH_ELEM(out_dtype, OT,
                       B200_CUDA_OK(launch_kernel(nsum == 1   ? dyt_residual_vec_kernel<OT, 1>
                                                  : nsum == 2 ? dyt_residual_vec_kernel<OT, 2>
                                                              : dyt_residual_vec_kernel<OT, 0>,
                                                  vec_grid(W / 4, th, T), dim3(th), 0, (cudaStream_t)stream, x,
                                                  y, nsum, y2, w1, b1, alpha1, w2, b2, alpha2, (OT*)out2, W, T)));
    return B200_OK;
  }
  B200_DISPATCH_ELEM(out_dtype, OT,
                     B200_CUDA_OK(launch_kernel(dyt_residual_kernel<OT>, dim3(flat_grid(total, 256)), dim3(256), 0,
                                                (cudaStream_t)stream, x, y, nsum, y2, w1, b1, alpha1, w2, b2, alpha2, (OT*)out2,
                                                W, total)));
  return B200_OK;
}

int b200_gated_group_rmsnorm(const float* y, const float* z, int ldz, const float* w, void* out, int out_dtype, int T,
                             int inner, int groups, float eps, void* stream) {
  B200_REQUIRE(y && z && w && out, "gated_group_rmsnorm: null pointer");
  B200_REQUIRE(groups >= 1 && inner % groups == 0, "gated_group_rmsnorm: %d channels do not split into %d groups", inner, groups);
  B200_REQUIRE((size_t)(inner / groups) * 4 <= 160 * 1024, "gated_group_rmsnorm: group of %d too wide", inner / groups);
  if (T <= 0) return B200_OK;
  const int gs = inner / groups, oes = out_dtype == B200_BF16 ? 2 : 4;
  const bool many = gs <= 128 || 5LL * T * groups >= 8LL * gs;
  if (many && gs % 4 == 0 && gs <= 1024 && groups <= 65535 && ldz % 4 == 0 && vec4_ok(y) && vec4_ok(z) && vec4_ok(w) && vec4_ok(out, oes)) {
    const int warps = T >= 8 * 148 ? 8 : 2;  // small batches spread over the SMs
#define GGR(V)                                                                                                                             \
  B200_DISPATCH_ELEM(out_dtype, OT,                                                                                                        \
                     B200_CUDA_OK(launch_kernel(gated_group_rmsnorm_warp_kernel<OT, V>, dim3((T + warps - 1) / warps, groups),             \
                                                dim3(32 * warps), 0, (cudaStream_t)stream, y, z, ldz, w, (OT*)out, inner, groups, eps, T)))
    if (gs <= 128) GGR(1);
    else if (gs <= 256) GGR(2);
    else if (gs <= 512) GGR(4);
    else GGR(8);
#undef GGR
    return B200_OK;
  }
  const size_t smem = (size_t)(inner / groups) * 4;
  B200_DISPATCH_ELEM(out_dtype, OT, {
    if (smem > 48 * 1024)
      B200_CUDA_OK(cudaFuncSetAttribute(gated_group_rmsnorm_kernel<OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    B200_CUDA_OK(launch_kernel(gated_group_rmsnorm_kernel<OT>, dim3(T, groups), dim3(256), smem, (cudaStream_t)stream, y, z, ldz,
                               w, (OT*)out, inner, groups, eps));
  });
  return B200_OK;
}

int b200_clamped_glu(const float* gate_up, void* out, int out_dtype, int T, int ff, float limit, void* stream) {
  B200_REQUIRE(gate_up && out, "clamped_glu: null pointer");
  if (T <= 0) return B200_OK;
  const int64_t total = (int64_t)T * ff;
  if (ff % 4 == 0 && vec4_ok(gate_up) && vec4_ok(out, out_dtype == B200_BF16 ? 2 : 4)) {
    const int th = vec_threads(ff / 4);
    B200_DISPATCH_ELEM(out_dtype, OT,
                       B200_CUDA_OK(launch_kernel(clamped_glu_vec_kernel<OT>, vec_grid(ff / 4, th, T), dim3(th), 0, (cudaStream_t)stream,
                                                  gate_up, (OT*)out, ff, limit, T)));
    return B200_OK;
  }
  B200_DISPATCH_ELEM(out_dtype, OT,
                     B200_CUDA_OK(launch_kernel(clamped_glu_kernel<OT>, dim3(flat_grid(total, 256)), dim3(256), 0,
                                                (cudaStream_t)stream, gate_up, (OT*)out, ff, limit, total)));
  return B200_OK;
}

}  // extern "C"
