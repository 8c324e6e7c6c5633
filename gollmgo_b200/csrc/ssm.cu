// A state-space layer of the Mamba-2 kind around the linear recurrence of delta_rule.cu.  Per head
// (P values, a state S [N, P] in float32 carried in the request's state slot):
//     S <- exp(-exp(A_log) dt) S + dt B x^T;   y = S^T C + D x
// with x (H heads of P values), B and C (G groups of N values; head h reads group h / (H / G)) passed
// through a short causal convolution per channel (with bias) and SiLU, dt = softplus(dt + dt_bias)
// per head.  The result is multiplied by silu(z) and RMS-normed in equal parts of the row.
//
// Kernels of a step (any mix of prompt portions and single decoded tokens):
//   ssm_prep   per (token, 128 channels): convolution + bias + SiLU from the projection's columns
//              [z | x | B | C | dt] and the window carried in the state slot; written as float32 rows
//              [C | B | x], the order the recurrence kernel reads (q, k, v); the last block of a token
//              computes the step size and the decay.  Then the window is moved on.
//   (the recurrence: gg_delta_recur with plain = 1: k = B, q = C, v = x, beta = dt)
//   ssm_out    per (token, part): (y + D x) * silu(z), divided by the part's root mean square, times
//              the weight
// Everything here is float32 arithmetic; the projection that comes in and the result that goes out
// are in the activation type.
#include "short_conv.cuh"

int conv_state_update(const void* x, long long x_stride, int dtype, float* conv_state, const int* cu_q_lens,
                      const int* context_lens, const int* state_slots, int B, int C, int taps, cudaStream_t stream);

__device__ __forceinline__ float ssm_silu(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float ssm_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

#define SSM_CH 128

// grid (T, ceil(Cc / 128) + 1).  proj [T, stride]: [z: inner | x: inner | B: G*N | C: G*N | dt: H];
// conv_w [Cc, taps], conv_b [Cc] over the channels x, B, C (Cc = inner + 2 G N); conv_state
// [slots, taps-1, Cc] holds the inputs at positions start-(taps-1) .. start-1 of the sequence.
template <typename TA>
__global__ void ssm_prep_kernel(const TA* __restrict__ proj, long long stride, const float* __restrict__ conv_w,
                                const float* __restrict__ conv_b, const float* __restrict__ conv_state,
                                const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                                const int* __restrict__ cu_q_lens, const int* __restrict__ context_lens,
                                const int* __restrict__ state_slots, int B, int H, int P, int G, int N, int taps,
                                float* __restrict__ cbx, float* __restrict__ dt_out, float* __restrict__ decay) {
  pdl_trigger();
  const int t = blockIdx.x;
  const int inner = H * P, GN = G * N, Cc = inner + 2 * GN;
  const int b = seq_of_token(cu_q_lens, B, t);
  const int t0 = cu_q_lens[b], qlen = cu_q_lens[b + 1] - t0;
  const int slot = state_slots[b];
  const int start = context_lens[b] - qlen;
  pdl_wait();
  if (blockIdx.y == gridDim.y - 1) {
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
      const float dt = ssm_softplus(to_f32(proj[(size_t)t * stride + 2 * inner + 2 * GN + h]) + dt_bias[h]);
      dt_out[(size_t)t * H + h] = dt;
      decay[(size_t)t * H + h] = expf(-expf(a_log[h]) * dt);
    }
    return;
  }
  const int c = blockIdx.y * SSM_CH + threadIdx.x;
  if (c >= Cc) return;
  const int i = t - t0;
  const float* st = (slot >= 0 && start > 0) ? conv_state + (size_t)slot * (taps - 1) * Cc : nullptr;
  float acc = conv_b ? conv_b[c] : 0.f;
  for (int j = 0; j < taps; ++j) {
    const int src = i - (taps - 1) + j;
    float xv;
    if (src >= 0) xv = to_f32(proj[(size_t)(t0 + src) * stride + inner + c]);
    else xv = st ? st[(size_t)(taps - 1 + src) * Cc + c] : 0.f;
    acc = fmaf(conv_w[(size_t)c * taps + j], xv, acc);
  }
  // x, B, C -> rows [C | B | x]
  const int dst = c < inner ? 2 * GN + c : (c < inner + GN ? GN + (c - inner) : c - inner - GN);
  cbx[(size_t)t * Cc + dst] = ssm_silu(acc);
}

// The same for TAPS taps and regions of whole groups of four channels: grid (tokens / per, groups of 128 threads + 1),
// four channels a thread (short_conv.cuh).  Bound by the latency of a block's dependent reads and by SiLU's exponential and division:
// 2048 tokens of 4352 channels take 18 us (bytes at the copy rate: 8), where the kernel above, which reads every row `taps`
// times two bytes a thread, takes 76.
template <typename TA, int TAPS>
__global__ void __launch_bounds__(CONV_THREADS, 8)
ssm_prep_vec_kernel(const TA* __restrict__ proj, long long stride, const float* __restrict__ conv_w, const float* __restrict__ conv_b,
                    float* conv_state, const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                    const int* __restrict__ cu_q_lens, const int* __restrict__ context_lens, const int* __restrict__ state_slots, int T,
                    int B, int H, int P, int G, int N, int per, int single, float* __restrict__ cbx, float* __restrict__ dt_out,
                    float* __restrict__ decay) {
  pdl_trigger();
  const int ta = blockIdx.x * per, tb = min(T, ta + per);
  const int inner = H * P, GN = G * N, Cc = inner + 2 * GN;
  if (blockIdx.y == gridDim.y - 1) {
    pdl_wait();
    for (int i = threadIdx.x; i < (tb - ta) * H; i += CONV_THREADS) {
      const int t = ta + i / H, h = i % H;
      const float dt = ssm_softplus(to_f32(proj[(size_t)t * stride + 2 * inner + 2 * GN + h]) + dt_bias[h]);
      dt_out[(size_t)t * H + h] = dt;
      decay[(size_t)t * H + h] = expf(-expf(a_log[h]) * dt);
    }
    return;
  }
  const int c = (blockIdx.y * CONV_THREADS + threadIdx.x) << 2;
  if (c >= Cc) return;
  const int dst = c < inner ? 2 * GN + c : (c < inner + GN ? GN + (c - inner) : c - inner - GN);    // rows [C | B | x]
  conv_tokens<TAPS>(proj + inner, stride, conv_w, conv_b, conv_state, cu_q_lens, context_lens, state_slots, B, Cc, c, ta, tb, single, true,
                    [&](int t, float4 y) { store4(cbx + (size_t)t * Cc + dst, y); });
}

// grid (T, parts): part p of token t covers inner / parts values.
template <typename TA>
__global__ void ssm_out_kernel(const float* __restrict__ y_raw, const float* __restrict__ cbx, int x_col, int Cc,
                               const TA* __restrict__ z, long long z_stride, const float* __restrict__ D,
                               const float* __restrict__ w, float eps, int P, int part, TA* __restrict__ out, int inner) {
  extern __shared__ float vals[];       // part floats + 33
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, c0 = blockIdx.y * part;
  float ss = 0.f;
  for (int e = threadIdx.x; e < part; e += blockDim.x) {
    const int c = c0 + e;
    const float x = cbx[(size_t)t * Cc + x_col + c];
    const float v = (y_raw[(size_t)t * inner + c] + D[c / P] * x) * ssm_silu(to_f32(z[(size_t)t * z_stride + c]));
    vals[e] = v;
    ss += v * v;
  }
  const float f = rsqrtf(block_sum(ss, vals + part) / (float)part + eps);
  for (int e = threadIdx.x; e < part; e += blockDim.x)
    out[(size_t)t * inner + c0 + e] = from_f32<TA>(vals[e] * f * w[c0 + e]);
}

// The same, four neighbouring values at a time and NV such groups a thread, kept in registers.  Bound by memory: 2048 tokens
// of 4096 values take 27 us (bytes at the copy rate: 15); a value at a time through shared memory 40.
template <typename TA, int NV>
__global__ void __launch_bounds__(1024)
ssm_out_vec_kernel(const float* __restrict__ y_raw, const float* __restrict__ cbx, int x_col, int Cc, const TA* __restrict__ z,
                   long long z_stride, const float* __restrict__ D, const float* __restrict__ w, float eps, int P, int part,
                   TA* __restrict__ out, int inner) {
  __shared__ float red[33];
  pdl_trigger();
  pdl_wait();
  const size_t t = blockIdx.x;
  const int c0 = blockIdx.y * part;
  float4 y[NV], x[NV], g[NV];
  float dh[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int e = (i * blockDim.x + threadIdx.x) << 2, c = c0 + e;
    if (e < part) {
      y[i] = load4(y_raw + t * inner + c);
      x[i] = load4(cbx + t * Cc + x_col + c);
      g[i] = load4(z + t * z_stride + c);
      dh[i] = D[c / P];
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (((i * blockDim.x + threadIdx.x) << 2) < part) {
      y[i].x = (y[i].x + dh[i] * x[i].x) * ssm_silu(g[i].x);
      y[i].y = (y[i].y + dh[i] * x[i].y) * ssm_silu(g[i].y);
      y[i].z = (y[i].z + dh[i] * x[i].z) * ssm_silu(g[i].z);
      y[i].w = (y[i].w + dh[i] * x[i].w) * ssm_silu(g[i].w);
      ss += y[i].x * y[i].x + y[i].y * y[i].y + (y[i].z * y[i].z + y[i].w * y[i].w);
    }
  const float f = rsqrtf(block_sum(ss, red) / (float)part + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int e = (i * blockDim.x + threadIdx.x) << 2, c = c0 + e;
    if (e < part) {
      const float4 ww = load4(w + c);
      store4(out + t * inner + c, make_float4(y[i].x * f * ww.x, y[i].y * f * ww.y, y[i].z * f * ww.z, y[i].w * f * ww.w));
    }
  }
}

extern "C" int gg_ssm_prep(const void* proj, long long stride, int dtype, const float* conv_w, const float* conv_b,
                           float* conv_state, const float* a_log, const float* dt_bias, const int* cu_q_lens,
                           const int* context_lens, const int* state_slots, int T, int B, int H, int P, int G, int N,
                           int taps, float* cbx, float* dt_out, float* decay, cudaStream_t stream) {
  GG_REQUIRE(T >= 0 && B > 0 && H > 0 && P > 0 && G > 0 && N > 0 && H % G == 0, "ssm_prep: bad sizes T=%d B=%d H=%d P=%d G=%d N=%d", T, B, H, P, G, N);
  GG_REQUIRE(taps >= 1 && taps <= 17, "ssm_prep: %d taps are outside 1..17", taps);
  const int inner = H * P, Cc = inner + 2 * G * N;
  GG_REQUIRE(stride >= (long long)inner + Cc + H, "ssm_prep: rows of %lld values are too short", stride);
  GG_REQUIRE(taps == 1 || conv_state, "ssm_prep: no room for the convolution's window");
  if (T == 0) return GG_OK;
  const int GN = G * N;
  if (taps >= 2 && taps <= 4 && inner % 4 == 0 && GN % 4 == 0 && stride % 4 == 0 && ((size_t)proj % 16) == 0 && ((size_t)conv_w % 16) == 0 &&
      (!conv_b || ((size_t)conv_b % 16) == 0) && ((size_t)conv_state % 16) == 0 && ((size_t)cbx % 16) == 0 && Cc / 4 / CONV_THREADS < 65000) {
    const int single = T == B, per = conv_tokens_a_block(T, B, (Cc / 4 + CONV_THREADS - 1) / CONV_THREADS);
    const dim3 vgrid((T + per - 1) / per, (Cc / 4 + CONV_THREADS - 1) / CONV_THREADS + 1);
#define SP_GO(TA, TAPS)                                                                                                              \
  gg_launch(ssm_prep_vec_kernel<TA, TAPS>, vgrid, dim3(CONV_THREADS), 0, stream, (const TA*)proj, stride, conv_w, conv_b, conv_state, a_log, \
            dt_bias, cu_q_lens, context_lens, state_slots, T, B, H, P, G, N, per, single, cbx, dt_out, decay)
#define SP_TAPS(TA) do { if (taps == 2) SP_GO(TA, 2); else if (taps == 3) SP_GO(TA, 3); else SP_GO(TA, 4); } while (0)
    if (dtype == GG_F32) SP_TAPS(float);
    else if (dtype == GG_BF16) SP_TAPS(__nv_bfloat16);
    else return gg_fail(GG_ERR_INVALID, "ssm_prep: unknown dtype %d", dtype);
#undef SP_TAPS
#undef SP_GO
    const int rc = gg_check_launch("ssm_prep");
    if (rc || single) return rc;
    return conv_state_update((const char*)proj + (size_t)inner * (dtype == GG_F32 ? 4 : 2), stride, dtype, conv_state, cu_q_lens,
                             context_lens, state_slots, B, Cc, taps, stream);
  }
  const dim3 grid(T, (Cc + SSM_CH - 1) / SSM_CH + 1);
  GG_REQUIRE(grid.y <= 65535, "ssm_prep: too many channels");
  if (dtype == GG_F32)
    gg_launch(ssm_prep_kernel<float>, grid, dim3(SSM_CH), 0, stream, (const float*)proj, stride, conv_w, conv_b, (const float*)conv_state, a_log, dt_bias, cu_q_lens, context_lens, state_slots, B, H, P, G, N, taps, cbx, dt_out, decay);
  else if (dtype == GG_BF16)
    gg_launch(ssm_prep_kernel<__nv_bfloat16>, grid, dim3(SSM_CH), 0, stream, (const __nv_bfloat16*)proj, stride, conv_w, conv_b, (const float*)conv_state, a_log, dt_bias, cu_q_lens, context_lens, state_slots, B, H, P, G, N, taps, cbx, dt_out, decay);
  else
    return gg_fail(GG_ERR_INVALID, "ssm_prep: unknown dtype %d", dtype);
  int rc = gg_check_launch("ssm_prep");
  if (rc || taps == 1) return rc;
  const size_t esize = dtype == GG_F32 ? 4 : 2;
  return conv_state_update((const char*)proj + (size_t)inner * esize, stride, dtype, conv_state, cu_q_lens, context_lens,
                           state_slots, B, Cc, taps, stream);
}

extern "C" int gg_ssm_out(const float* y_raw, const float* cbx, int x_col, int Cc, const void* z, long long z_stride,
                          int dtype, const float* D, const float* w, float eps, int T, int H, int P, int parts, void* out,
                          cudaStream_t stream) {
  GG_REQUIRE(T >= 0 && H > 0 && P > 0 && parts > 0 && (H * P) % parts == 0 && parts <= 65535, "ssm_out: bad sizes T=%d H=%d P=%d parts=%d", T, H, P, parts);
  if (T == 0) return GG_OK;
  const int inner = H * P, part = inner / parts;
  if (part % 4 == 0 && P % 4 == 0 && part <= 16384 && x_col % 4 == 0 && Cc % 4 == 0 && z_stride % 4 == 0 && ((size_t)y_raw % 16) == 0 &&
      ((size_t)cbx % 16) == 0 && ((size_t)z % 16) == 0 && ((size_t)w % 16) == 0 && ((size_t)out % 16) == 0 &&
      (dtype == GG_F32 || dtype == GG_BF16)) {
    // few rows (decoded tokens): one group of four a thread, so that a row is as many threads as there are; else four,
    // whose loads are all on their way together
    const int nv = part <= 4096 && (long long)T * parts <= 2 * 148 ? 1 : 4;
    const dim3 vgrid(T, parts), block(((part / 4 + nv - 1) / nv + 31) / 32 * 32);
#define SO_GO(TA, NV) \
  gg_launch(ssm_out_vec_kernel<TA, NV>, vgrid, block, 0, stream, y_raw, cbx, x_col, Cc, (const TA*)z, z_stride, D, w, eps, P, part, (TA*)out, inner)
    if (dtype == GG_F32) { if (nv == 1) SO_GO(float, 1); else SO_GO(float, 4); }
    else { if (nv == 1) SO_GO(__nv_bfloat16, 1); else SO_GO(__nv_bfloat16, 4); }
#undef SO_GO
    return gg_check_launch("ssm_out");
  }
  const size_t smem = (size_t)(part + 33) * sizeof(float);
  GG_REQUIRE(smem <= 200 * 1024, "ssm_out: parts of %d values do not fit in shared memory", part);
  // four values a thread where the part is long: a step of few decoded tokens has T * parts blocks and waits on
  // each thread's chain of reads
  const int threads = part >= 4096 ? 1024 : (part >= 2048 ? 512 : (part >= 1024 ? 256 : (part >= 256 ? 128 : 64)));
  const dim3 grid(T, parts);
  cudaError_t e = cudaSuccess;
  if (dtype == GG_F32) {
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(ssm_out_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "ssm_out: %s", cudaGetErrorString(e));
    gg_launch(ssm_out_kernel<float>, grid, dim3(threads), smem, stream, y_raw, cbx, x_col, Cc, (const float*)z, z_stride, D, w, eps, P, part, (float*)out, inner);
  } else if (dtype == GG_BF16) {
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(ssm_out_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "ssm_out: %s", cudaGetErrorString(e));
    gg_launch(ssm_out_kernel<__nv_bfloat16>, grid, dim3(threads), smem, stream, y_raw, cbx, x_col, Cc, (const __nv_bfloat16*)z, z_stride, D, w, eps, P, part, (__nv_bfloat16*)out, inner);
  } else
    return gg_fail(GG_ERR_INVALID, "ssm_out: unknown dtype %d", dtype);
  return gg_check_launch("ssm_out");
}
