// The gated delta rule (delta_rule.cu) over prompt portions in chunks.  Inside a chunk, with the state S [d, dv] before it and
// G_i = g_1 .. g_i, the token's writes u_i solve a unit lower triangular system:
//     u_i = b_i (v_i - G_i S^T k_i - sum_(j<i) (G_i / G_j) (k_i . k_j) u_j)
// so with A_ij = b_i (G_i / G_j) (k_i . k_j) below the diagonal, U = (I + A)^-1 (b V) - (I + A)^-1 (b G K) S = V' - W S.
//   delta_solve   all chunks of 64 tokens at once: W and V', by forward substitution, two columns of [b G K | b V] a thread
//   delta_states  per (sequence, head, 16 value columns), one chunk after the other: U = V' - W S, S <- G_n S + sum_j (G_n / G_j)
//                 k_j u_j^T; leaves S before every 128 tokens for the rows
//   linear_rows   all chunks of 128 tokens at once (linear_chunks.cu): o_i = G_i S^T q_i + sum_(j<=i) (G_i / G_j) (q_i . k_j) u_j
// The first two run on mma.sync: a token's write needs the state before it, so what can run beside one another is small (16 value
// columns of a head, 64 tokens), and the operands go from one product's sums to the next one's in registers.  Products are float32
// ones made of three tf32 ones, as in linear_chunks.cu; the ratios come from float64 sums of logarithms; the state is float32.
// Measured (B200), 1280 + 768 tokens, 16 heads 128 x 128 on 4 of q and k: 35 + 75 + 48 us, token by token 312.  What bounds them: the
// solving, issue slots (splitting operands, 0.5 instructions a clock and scheduler) and the waits between its steps; the states, the
// tensor cores' rate on mma.sync tf32 (2.5 clocks a product: 1930 of some 3250 clocks a chunk and group) and the exchange of sums.
// A row of (I + A)^-1 is a product of contractions (I - b k k^T, k a unit vector), so solving does not grow errors.
// Waits on barriers are bounded; one that runs out sets *status.
#include "delta_chunks.cuh"
#include "tc_common.cuh"

enum { DC_ERR_WAIT = 91 };

#define DC_C 64                // tokens of a chunk
#define DC_WARPS 8             // of delta_states
#define DC_COLS 16             // value columns of one CTA of delta_states
#define DC_AP (DC_C + 4)
#define DC_HEADS 4             // most heads of one block of delta_solve

__device__ __forceinline__ void dc_cp16(float* dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void dc_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void dc_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// c += a b, 16 x 8 x 8 tf32.  A thread (r = lane / 4, q = lane % 4) has of a: (r, k = q), (r + 8, q), (r, q + 4), (r + 8, q + 4);
// of b: (k = q, n = r), (q + 4, r); of c: (r, n = 2 q), (r, 2 q + 1), (r + 8, 2 q), (r + 8, 2 q + 1).  Which value of the inner
// dimension is called which k is free: with n = 2 q called k = q and n = 2 q + 1 called q + 4, sums c are the next product's a.
__device__ __forceinline__ void dc_mma(float (&c)[4], const float (&a)[4], float b0, float b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                 "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}
// x = hi + lo, hi to 11 bits
__device__ __forceinline__ void dc_split(float x, float& hi, float& lo) {
  hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
  lo = x - hi;
}
// sums c as the next product's a
__device__ __forceinline__ void dc_split_sums(const float (&c)[4], float (&hi)[4], float (&lo)[4]) {
  dc_split(c[0], hi[0], lo[0]); dc_split(c[2], hi[1], lo[1]); dc_split(c[1], hi[2], lo[2]); dc_split(c[3], hi[3], lo[3]);
}
// main gets hi hi, small and less the other two (chains of their own)
__device__ __forceinline__ void dc_mma3(float (&main)[4], float (&small)[4], float (&less)[4], const float (&ahi)[4], const float (&alo)[4], float b0, float b1) {
  float h0, l0, h1, l1;
  dc_split(b0, h0, l0);
  dc_split(b1, h1, l1);
  dc_mma(small, alo, h0, h1);
  dc_mma(main, ahi, h0, h1);
  dc_mma(less, ahi, l0, l1);
}

// log2 of a decay; one of 0 (its exponential underflowed) stays finite and still wipes out what came before.  NaN stays NaN.
__device__ __forceinline__ float dc_log2(float g) {
  const float l = log2f(g);
  return l < -2000.f ? -2000.f : l;
}

// ---------------------------------------------------------------- the triangular systems
// grid (2 tiles, H / heads), 256 threads: a chunk of `heads` heads that share k.  The products k_i . k_j once; then per head -A, the
// inverses of its 8 x 8 blocks on the diagonal, and the columns of [b G K | b V], sixteen a tile, two tiles a warp at a time: a block
// of eight tokens is final once its inverse has met it, and leaves the blocks below with one product each.
template <int D>
__global__ void __launch_bounds__(256, 2)
delta_solve_kernel(const DeltaChunkArgs p) {
  extern __shared__ __align__(16) float dc_sm[];
  constexpr int KP = D + 4;
  float* ks = dc_sm;                                   // [64][KP]
  float* gs = ks + DC_C * KP;                          // [i][DC_AP]: k_i . k_j
  float* at = gs + DC_C * DC_AP;                       // [i][DC_AP]: -A_ij
  float* ts = at + DC_C * DC_AP;                       // [8][8][8]: the inverses
  float* vs = ts + 8 * 64;                             // [64][VP]: v of the head at hand
  __shared__ float2 L[DC_HEADS][DC_C];                 // sums of the logarithms, in two parts
  __shared__ float bs[DC_HEADS][DC_C], bg[DC_HEADS][DC_C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, q = lane & 3, h0 = blockIdx.y * p.heads;
  const int b = p.tile_seq[blockIdx.x >> 1], q0 = p.tile_q0[blockIdx.x >> 1] + DC_C * (blockIdx.x & 1);
  const int qlen = p.cu_q_lens[b + 1] - p.cu_q_lens[b], t0 = p.cu_q_lens[b] + q0, n = min(DC_C, qlen - q0), d = p.d;
  const int VP = p.dv + 4, vper = p.dv >> 2;
  pdl_trigger();
  pdl_wait();
  if (n <= 0) return;
  auto fetch_v = [&](int h) {
    const float* vr = p.rows + (size_t)t0 * p.row_stride + p.v_col + (size_t)h * p.dv;
    for (int e = tid; e < DC_C * vper; e += 256) {
      const int t = e / vper, c = (e - t * vper) << 2;
      dc_cp16(vs + t * VP + c, t < n ? vr + (size_t)t * p.row_stride + c : vr, t < n);
    }
    dc_commit();
  };
  const float* kr = p.rows + (size_t)t0 * p.row_stride + p.k_col + (size_t)(h0 / (p.H / p.G)) * d;
  for (int e = tid; e < DC_C * (D / 4); e += 256) {
    const int t = e / (D / 4), c = (e % (D / 4)) << 2;
    const bool there = t < n && c < d;
    dc_cp16(ks + t * KP + c, there ? kr + (size_t)t * p.row_stride + c : kr, there);
  }
  dc_commit();
  fetch_v(h0);
  if (warp < p.heads) {                                // sums of the logarithms: two tokens a lane
    const int h = h0 + warp;
    double a[2], s = 0.0;
    float f[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = 2 * lane + i;
      const size_t at_j = (size_t)(t0 + j) * p.H + h;
      s += (double)(j < n ? dc_log2(p.decay[at_j]) : 0.f);
      a[i] = s;
      f[i] = j < n ? p.beta[at_j] : 0.f;
    }
    double incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    double before = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) before = 0.0;                       // (not incl - s: a NaN would reach the lane's tokens before it)
    const double all = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = 2 * lane + i;
      const double l = before + a[i];
      L[warp][j] = make_float2((float)l, (float)(l - (double)(float)l));
      bs[warp][j] = f[i];
      bg[warp][j] = f[i] * exp2f((float)l);
      if (j < n) p.tail[(size_t)(t0 + j) * p.H + h] = exp2f((float)(all - l));
    }
    if (lane == 0) p.factor[(size_t)blockIdx.x * p.H + h] = exp2f((float)all);
  }
  dc_wait<1>();
  __syncthreads();
  constexpr int DW = D / DC_WARPS, NT = DW / 8;
  if (h0 % (p.H / p.G) == 0) {                         // K as delta_states reads it: (warp, 8 tokens, q, r): tokens 2 q, 2 q + 1, NT values each
    float* o = p.k + ((size_t)blockIdx.x * p.G + h0 / (p.H / p.G)) * DC_C * D;
    for (int e = tid; e < DC_C * D / (2 * NT); e += 256) {
      const int lr = e & 7, lq = e >> 3 & 3, k = e >> 5 & 7, w = e >> 8;
      const float* at_k = ks + (8 * k + 2 * lq) * KP + w * DW + NT * lr;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int t = 0; t < NT; ++t) o[e * 2 * NT + i * NT + t] = at_k[i * KP + t];
    }
  }
  for (int tile = warp; tile < 20; tile += 8) {        // k_i . k_j: sixteen i, eight j a tile, those that reach below the diagonal
    const int rb = tile < 2 ? 0 : tile < 6 ? 1 : tile < 12 ? 2 : 3, nb = tile - rb * (rb + 1);
    float main[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f}, less[4] = {0.f, 0.f, 0.f, 0.f};
    const float* ka = ks + (16 * rb + r) * KP + 8 * q;
    const float* kb = ks + (8 * nb + r) * KP + 8 * q;
#pragma unroll
    for (int e = 0; e < D; e += 32) {                  // 32 values of d in four steps: q has 8 q .. 8 q + 7
      float x[4][4], y[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        *reinterpret_cast<float4*>(x[2 * u]) = *reinterpret_cast<const float4*>(ka + e + 4 * u);
        *reinterpret_cast<float4*>(x[2 * u + 1]) = *reinterpret_cast<const float4*>(ka + 8 * KP + e + 4 * u);
        *reinterpret_cast<float4*>(y[u]) = *reinterpret_cast<const float4*>(kb + e + 4 * u);
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float hi[4], lo[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) dc_split(x[u][t], hi[u], lo[u]);
        dc_mma3(main, small, less, hi, lo, y[0][t], y[1][t]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) main[e] += small[e] + less[e];
    float* o = gs + (16 * rb + r) * DC_AP + 8 * nb + 2 * q;
    *reinterpret_cast<float2*>(o) = make_float2(main[0], main[1]);
    *reinterpret_cast<float2*>(o + 8 * DC_AP) = make_float2(main[2], main[3]);
  }
  __syncthreads();
  const int nk = D / 16, tiles = nk + p.dv / 16;
  for (int hh = 0; hh < p.heads; ++hh) {
    const int h = h0 + hh;
    for (int e = tid; e < DC_C * DC_C; e += 256) {     // (the rest is never read)
      const int i = e / DC_C, j = e % DC_C;
      const float2 li = L[hh][i], lj = L[hh][j];
      if (j < i) at[i * DC_AP + j] = -(bs[hh][i] * exp2f((li.x - lj.x) + (li.y - lj.y)) * gs[i * DC_AP + j]);
    }
    __syncthreads();
    if (tid < DC_C) {                                  // column c of the inverse of block k
      const int k = tid >> 3, c = tid & 7;
      const float* a = at + 8 * k * DC_AP + 8 * k;
      float t[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float v = i == c ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < i; ++j)
          if (j >= c) v = fmaf(a[i * DC_AP + j], t[j], v);
        t[i] = v;
        ts[k * 64 + i * 8 + c] = v;
      }
    }
    dc_wait<0>();
    __syncthreads();
    float* u = p.o_raw + ((size_t)t0 * p.H + h) * p.dv;
    float* w = p.w + ((size_t)blockIdx.x * p.H + h) * DC_C * D;       // [warp][token][DW]
    for (int m0 = warp; m0 < tiles; m0 += 16) {
      float x[2][8][4];                                // [tile][tokens 8 j ..]: (column r, token 2 q), (r, 2 q + 1), (r + 8, 2 q), ..
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int mt = m0 + 8 * m;
        const bool key = mt < nk;
        const int c = key ? 16 * mt + r : 16 * (mt - nk) + r;
        const bool there = mt < tiles;                 // (columns of K past d are zeros)
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int t = 8 * j + 2 * q + e;
            const float* src = key ? ks + t * KP + c : vs + t * VP + c;
            const float f = key ? bg[hh][t] : bs[hh][t];
            x[m][j][e] = there ? src[0] * f : 0.f;
            x[m][j][2 + e] = there ? src[8] * f : 0.f;
          }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float hi[2][4], lo[2][4];
        const float2 tb = *reinterpret_cast<const float2*>(ts + j * 64 + r * 8 + 2 * q);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          float (&y)[4] = x[m][j];
          // the inverse's zeros above the diagonal would carry a bad value to the tokens before it
          float z = 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) z = fmaf(y[e], 0.f, z);
          if (__any_sync(0xffffffffu, !(z == 0.f))) {
            const float* a = at + (8 * j + 2 * q) * DC_AP + 8 * j;
#pragma unroll 1
            for (int s = 0; s < 8; ++s) {
              const int from = (lane & ~3) | (s >> 1);
              const float v0 = __shfl_sync(0xffffffffu, s & 1 ? y[1] : y[0], from), v1 = __shfl_sync(0xffffffffu, s & 1 ? y[3] : y[2], from);
              if (2 * q > s) { y[0] = fmaf(a[s], v0, y[0]); y[2] = fmaf(a[s], v1, y[2]); }
              if (2 * q + 1 > s) { y[1] = fmaf(a[DC_AP + s], v0, y[1]); y[3] = fmaf(a[DC_AP + s], v1, y[3]); }
            }
          } else {
            float main[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f}, less[4] = {0.f, 0.f, 0.f, 0.f};
            dc_split_sums(y, hi[m], lo[m]);
            dc_mma3(main, small, less, hi[m], lo[m], tb.x, tb.y);
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = main[e] + (small[e] + less[e]);
          }
          dc_split_sums(y, hi[m], lo[m]);
        }
#pragma unroll
        for (int i = j + 1; i < 8; ++i) {
          const float2 a = *reinterpret_cast<const float2*>(at + (8 * i + r) * DC_AP + 8 * j + 2 * q);
          float a0, a0l, a1, a1l;
          dc_split(a.x, a0, a0l);
          dc_split(a.y, a1, a1l);
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            dc_mma(x[m][i], lo[m], a0, a1);
            dc_mma(x[m][i], hi[m], a0l, a1l);
            dc_mma(x[m][i], hi[m], a0, a1);
          }
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int mt = m0 + 8 * m;
        const bool key = mt < nk;
        const int c = key ? 16 * mt + r : 16 * (mt - nk) + r;
        if (mt >= tiles) continue;
        float* o = key ? w + (DW == 16 ? mt : 2 * mt) * DC_C * DW + r : u + c;
        const size_t pitch = key ? DW : (size_t)p.H * p.dv, eight = key && DW == 8 ? DC_C * DW : 8;      // eight: to column c + 8
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int t = 8 * j + 2 * q + e;
            if (key || t < n) {
              o[(size_t)t * pitch] = x[m][j][e];
              o[(size_t)t * pitch + eight] = x[m][j][2 + e];
            }
          }
      }
    }
    __syncthreads();
    if (hh + 1 < p.heads) fetch_v(h + 1);
  }
}

// ---------------------------------------------------------------- the states, one chunk after the other
// grid (dv / 16 / NG, H, B), eight warps a group.  A group has sixteen columns: S^T, sixteen by d, stays in registers as the sums it was
// made by, an eighth of d a warp.  Per chunk: every warp's share of S^T W^T for all 64 tokens (the shares meet in shared memory, eight
// tokens a warp), U^T as the next product's operand to all warps, U^T K for the warp's part of d.  W and K of a chunk, 64 KB for keys
// of 128, come in one copy each, a chunk ahead; two groups share them and fill each other's waits.
template <int D, int NG>
__global__ void __launch_bounds__(NG * DC_WARPS * 32, 1)
delta_states_kernel(const DeltaChunkArgs p) {
  extern __shared__ __align__(16) float dc_sm[];
  constexpr int DW = D / DC_WARPS, NT = DW / 8;        // a warp's d: 2 NT neighbouring ones a q; tile t, column c of it: NT c + t
  constexpr int TILE = DC_C * D;
  float* wk = dc_sm;                                   // [2 stages][W, K][TILE]
  __shared__ int first_s, abort_s;
  __shared__ __align__(8) unsigned long long bars[4];  // [2] there, [2] used
  const int b = blockIdx.z, h = blockIdx.y, tid = threadIdx.x;
  const int slot = p.state_slots[b], s0 = p.cu_q_lens[b], qlen = p.cu_q_lens[b + 1] - s0;
  const unsigned there0 = tc_smem(&bars[0]), used0 = tc_smem(&bars[2]);
  if (tid == 0) {
    first_s = -1;
    abort_s = 0;
    for (int i = 0; i < 2; ++i) { mbar_init(there0 + 8 * i, 1); mbar_init(used0 + 8 * i, NG * DC_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  for (int i = tid; i < p.tiles; i += NG * DC_WARPS * 32)          // the sequence's first tile
    if (p.tile_seq[i] == b && p.tile_q0[i] == 0) first_s = i;
  __syncthreads();
  const int first = first_s;
  if (slot < 0 || first < 0) { pdl_trigger(); pdl_wait(); return; }
  const bool carry = p.context_lens[b] - qlen > 0;
  const int group = tid >> 8, warp = tid >> 5 & 7, lane = tid & 31, r = lane >> 2, q = lane & 3, d = p.d;
  const int col0 = (blockIdx.x * NG + group) * DC_COLS;
  float4* part = reinterpret_cast<float4*>(dc_sm + 4 * TILE) + group * (DC_WARPS * DC_WARPS + 8) * 32;     // [receiver][giver][lane]
  float4* uf = part + DC_WARPS * DC_WARPS * 32;        // [8 tokens][lane]
  const int chunks = (qlen + DC_C - 1) / DC_C;
  const size_t upitch = (size_t)p.H * p.dv;
  const int dq = warp * DW + 2 * NT * q;               // this thread's first d
  const bool has = dq < d;                             // (d is a multiple of 32)
  const size_t srow = (size_t)(col0 + r) * d + dq;     // in a head's state: column r; column r + 8 is 8 d further
  float* shead = p.state + ((size_t)slot * p.H + h) * p.dv * d + srow;
  float* ur = p.o_raw + ((size_t)(s0 + 8 * warp + 2 * q) * p.H + h) * p.dv + col0 + r;
  const float* tails = p.tail + (size_t)(s0 + 8 * warp + 2 * q) * p.H + h;
  const float* factors = p.factor + (size_t)(2 * first) * p.H + h;
  int left = qlen - 8 * warp - 2 * q;                  // tokens from this thread's first one of the chunk on
  pdl_wait();
  bool ok = true;
  auto wait = [&](unsigned bar, unsigned parity) {     // one that runs out: the chunks end here
    ok = ok && mbar_wait(bar, parity) && !*(volatile int*)&abort_s;
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) { atomicExch(p.status, DC_ERR_WAIT); atomicExch(&abort_s, 1); }
  };
  auto fetch = [&](int c) {                            // by one thread
    const float* src[2] = {p.w + ((size_t)(2 * first + c) * p.H + h) * TILE, p.k + ((size_t)(2 * first + c) * p.G + h / (p.H / p.G)) * TILE};
    mbar_expect_tx(there0 + 8 * (c & 1), 2 * TILE * 4);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(tc_smem(wk + (2 * (c & 1) + i) * TILE)), "l"(src[i]), "r"(TILE * 4), "r"(there0 + 8 * (c & 1)) : "memory");
  };
  if (tid == 0) fetch(0);
  // of a chunk's U this warp has tokens 8 warp .. + 7, a thread (columns r and r + 8) 8 warp + 2 q + e
  float vn[4], tn[2], fn = 0.f;
  auto ahead = [&] {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const bool there = left > e;
      vn[e] = there ? ur[e * upitch] : 0.f;
      vn[2 + e] = there ? ur[e * upitch + 8] : 0.f;
      tn[e] = there ? tails[e * p.H] : 0.f;
    }
    fn = *factors;
  };
  ahead();
  float S[NT][4];                                      // tile t: (column r, d = dq + t), (r, dq + NT + t), (r + 8, ..), (r + 8, ..)
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int t = 0; t < NT; ++t) S[t][2 * x + e] = carry && has ? shead[(size_t)(8 * x) * d + NT * e + t] : 0.f;
  auto save = [&](float* o) {                          // o: this thread's place in a head's state
    if (!has) return;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float* to = o + (size_t)(8 * x) * d + NT * e;
        if constexpr (NT == 2) *reinterpret_cast<float2*>(to) = make_float2(S[0][2 * x + e], S[1][2 * x + e]);
        else *to = S[0][2 * x + e];
      }
  };
  auto meet = [&] { asm volatile("bar.sync %0, 256;" ::"r"(1 + group) : "memory"); };      // the group's warps
  const unsigned char* wb = reinterpret_cast<const unsigned char*>(wk + (warp * DC_C + r) * DW + 2 * NT * q);
  const unsigned char* kb = reinterpret_cast<const unsigned char*>(wk + TILE + ((warp * 8 * 4 + q) * 8 + r) * 2 * NT);
  auto load = [&](float (&y)[2 * NT], const unsigned char* from, int k) {
    if constexpr (NT == 2) *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(from + k * 256 * NT);
    else *reinterpret_cast<float2*>(y) = *reinterpret_cast<const float2*>(from + k * 256 * NT);
  };
  for (int c = 0; c < chunks; ++c) {
    // (a wait that ran out: the loop goes on, without copies, to its end)
    if (tid < 32) {
      if (c > 0) wait(used0 + 8 * ((c + 1) & 1), ((c - 1) >> 1) & 1);
      if (ok && lane == 0 && c + 1 < chunks) fetch(c + 1);
    }
    const int stage = (c & 1) * 2 * TILE * 4;
    if ((c & 1) == 0 && (c > 0 || carry))              // the state before these 128 tokens (else nobody reads it)
      save(p.scratch + ((size_t)(first + (c >> 1)) * p.H + h) * p.dv * d + srow);
    {
      float hi[NT][4], lo[NT][4];
#pragma unroll
      for (int t = 0; t < NT; ++t) dc_split_sums(S[t], hi[t], lo[t]);
      wait(there0 + 8 * (c & 1), (c >> 1) & 1);
#pragma unroll
      for (int k = 0; k < 8; ++k) {                    // tokens 8 k ..
        float y[2 * NT];
        load(y, wb + stage, k);
        float main[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f}, less[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int t = 0; t < NT; ++t) dc_mma3(main, small, less, hi[t], lo[t], y[t], y[NT + t]);
#pragma unroll
        for (int e = 0; e < 4; ++e) main[e] += small[e] + less[e];
        part[(k * DC_WARPS + warp) * 32 + lane] = make_float4(main[0], main[1], main[2], main[3]);
      }
    }
    meet();
    {
      float4 v[DC_WARPS];
#pragma unroll
      for (int o = 0; o < DC_WARPS; ++o) v[o] = part[(warp * DC_WARPS + o) * 32 + lane];
#pragma unroll
      for (int o = 1; o < DC_WARPS; o *= 2)
#pragma unroll
        for (int i = 0; i < DC_WARPS; i += 2 * o) {
          v[i].x += v[i + o].x; v[i].y += v[i + o].y; v[i].z += v[i + o].z; v[i].w += v[i + o].w;
        }
      const float sum[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
      float keep[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool there = left > (e & 1);
        const float u = vn[e] - sum[e];
        if (there) ur[(e & 1) * upitch + (e >> 1) * 8] = u;
        keep[e] = there ? u * tn[e & 1] : 0.f;
      }
      uf[warp * 32 + lane] = make_float4(keep[0], keep[1], keep[2], keep[3]);
    }
    const float factor = fn;
    ur += DC_C * upitch;
    tails += DC_C * p.H;
    left -= DC_C;
    if (c + 1 < chunks) { factors += p.H; ahead(); }
    meet();
    {
      float main[NT][4], small[NT][4], less[NT][4];
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) main[t][e] = small[t][e] = less[t][e] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {                    // tokens 8 k ..
        float u[4], hi[4], lo[4], y[2 * NT];
        *reinterpret_cast<float4*>(u) = uf[k * 32 + lane];
        load(y, kb + stage, k);
        dc_split_sums(u, hi, lo);
#pragma unroll
        for (int t = 0; t < NT; ++t) dc_mma3(main[t], small[t], less[t], hi, lo, y[t], y[NT + t]);
      }
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[t][e] = fmaf(factor, S[t][e], main[t][e] + (small[t][e] + less[t][e]));
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(used0 + 8 * (c & 1));
  }
  pdl_trigger();                                       // only now: blocks of the next kernel that wait on a multiprocessor take room there
  save(shead);
}

// ---------------------------------------------------------------- launcher
template <int D, int NG> static int dc_states(const DeltaChunkArgs& p, cudaStream_t stream) {
  const size_t smem = 4 * DC_C * D * sizeof(float) + NG * (DC_WARPS * DC_WARPS + 8) * 32 * sizeof(float4);
  cudaError_t e = cudaFuncSetAttribute(delta_states_kernel<D, NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "delta_chunks: %s", cudaGetErrorString(e));
  gg_launch_after(delta_states_kernel<D, NG>, dim3(p.dv / DC_COLS / NG, p.H, p.B), dim3(NG * DC_WARPS * 32), smem, stream, p);
  return gg_check_launch("delta_states");
}

template <int D> static int dc_run(DeltaChunkArgs p, cudaStream_t stream) {
  constexpr int P = D + 4;
  const size_t solve = (DC_C * P + 2 * DC_C * DC_AP + 8 * 64 + DC_C * (p.dv + 4)) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(delta_solve_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solve);
  if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "delta_chunks: %s", cudaGetErrorString(e));
  // as many heads of a group a block as leave a block for every multiprocessor
  p.heads = 1;
  while (p.heads < DC_HEADS && p.H / p.G % (2 * p.heads) == 0 && 2ll * p.tiles * (p.H / (2 * p.heads)) >= 3 * 148 / 2) p.heads *= 2;
  gg_launch(delta_solve_kernel<D>, dim3(2 * p.tiles, p.H / p.heads), dim3(256), solve, stream, p);
  const int rc = gg_check_launch("delta_solve");
  if (rc) return rc;
  // two groups of columns a block where that leaves a block for most multiprocessors (one group alone waits half its time)
  return p.dv % (2 * DC_COLS) == 0 && (long long)p.B * p.H * (p.dv / (2 * DC_COLS)) >= 64 ? dc_states<D, 2>(p, stream) : dc_states<D, 1>(p, stream);
}

// gg_delta_recur (a decay per head) over the sequences whose chunks of 128 tokens are the tiles (all chunks of a sequence, in their
// order); the others are left alone.  Returns GG_ERR_UNSUPPORTED, and launches nothing, where sizes or addresses are not for
// these kernels.  Scratch the caller provides: float[num_tiles * H * (d * dv + 4)] and float[num_tiles * 128 * (H + G) * D + T * H]
// with D = 64 or 128, the first that holds d.
extern "C" int gg_delta_chunks(const float* qkv, const float* beta, const float* decay, float* state, float* scratch,
                               long long scratch_floats, float* w, long long w_floats, const int* tile_seq, const int* tile_q0,
                               int num_tiles, const int* cu_q_lens, const int* context_lens, const int* state_slots, int T, int B,
                               int G, int H, int d, int dv, float* o_raw, int* status, cudaStream_t stream) {
  GG_REQUIRE(T >= 0 && B > 0 && G > 0 && H > 0 && H % G == 0 && d > 0 && dv > 0 && num_tiles >= 0, "delta_chunks: bad sizes T=%d B=%d G=%d H=%d d=%d dv=%d", T, B, G, H, d, dv);
  GG_REQUIRE(qkv && beta && decay && state && scratch && w && o_raw && status, "delta_chunks: a pointer is null");
  DeltaChunkArgs p = {};
  p.rows = qkv; p.row_stride = 2ll * G * d + (long long)H * dv; p.k_col = G * d; p.v_col = 2 * G * d;
  p.beta = beta; p.decay = decay; p.state = state; p.scratch = scratch; p.o_raw = o_raw;
  const int D = d <= 64 ? 64 : 128;
  p.w = w; p.k = w + (size_t)num_tiles * 128 * H * D; p.tail = p.k + (size_t)num_tiles * 128 * G * D;
  p.factor = scratch + (size_t)num_tiles * H * d * dv;             // (two a tile; linear_rows has none of its own here)
  p.tile_seq = tile_seq; p.tile_q0 = tile_q0; p.tiles = num_tiles; p.cu_q_lens = cu_q_lens; p.context_lens = context_lens;
  p.state_slots = state_slots; p.T = T; p.B = B; p.G = G; p.H = H; p.d = d; p.dv = dv; p.status = status;
  if (d > 128 || d % 32 || dv % DC_COLS || dv > 256 || H > 65535 || B > 65535 || ((size_t)w % 16) || !delta_rows_supported(p)) return GG_ERR_UNSUPPORTED;
  GG_REQUIRE(scratch_floats >= (long long)num_tiles * H * ((long long)d * dv + 4) && w_floats >= num_tiles * 128ll * (H + G) * D + (long long)T * H,
             "delta_chunks: scratch of %lld and %lld values is too small", scratch_floats, w_floats);
  if (num_tiles == 0) return GG_OK;
  const int rc = d <= 64 ? dc_run<64>(p, stream) : dc_run<128>(p, stream);
  return rc ? rc : delta_rows(p, stream);
}
