// The gated delta rule (delta_rule.cu) over prompt portions in chunks of 64 tokens.  Inside a chunk, with the state S [d, dv] before
// it and G_i = g_1 .. g_i, the token's writes u_i solve a unit lower triangular system:
//     u_i = b_i (v_i - G_i S^T k_i - sum_(j<i) (G_i / G_j) (k_i . k_j) u_j)
// so with A_ij = b_i (G_i / G_j) (k_i . k_j) below the diagonal, U = (I + A)^-1 (b V) - (I + A)^-1 (b G K) S = V' - W S.
//   delta_solve   all chunks at once: W and V' by forward substitution, two columns of [b G K | b V] a thread
//   delta_states  per (sequence, head, 16 value columns), one chunk after the other: U = V' - W S, S <- G_n S + sum_j (G_n / G_j)
//                 k_j u_j^T; leaves S before every chunk for the rows
//   delta_rows    all chunks at once: o_i = G_i S^T q_i + sum_(j<=i) (G_i / G_j) (q_i . k_j) u_j
// All of it is float32 arithmetic, as in the walk over the tokens; sums of logarithms are float64.  The chunks' sums are short chains
// (8 or 16 terms, then a tree or a second sum).  Against float64, 40 steps of 320 to 2048 tokens, 16 and 32 heads: rows 1.1e-7 to
// 1.8e-7 (the walk 1.0e-7 to 3.3e-7; 0.56 to 1.09 of its), states 1.0e-7 to 1.9e-7 (1.3e-7 to 4.3e-7; 0.42 to 0.76 of its).  The same
// from three tf32 products a term: rows 6e-7 to 9e-7, states 5e-7 to 7e-7.  That is no faster where it counts: a multiprocessor does 128
// float32 multiply-adds a clock, and three tf32 mma.sync of 1024, 2.5 clocks each, 136.
// Measured (B200), 1280 + 768 tokens, 16 heads 128 x 128 on 4 of q and k: 35 + 84 + 52 us (token by token 312, with tf32 products 147).
// A row of (I + A)^-1 is a product of contractions (I - b k k^T, k a unit vector), so solving does not grow errors.
// Infinities and NaN reach the rows and states that they reach token by token, no earlier token.
// Waits on barriers are bounded; one that runs out sets *status, and the block waits (as long again) for its copies before it ends.
#include "tc_common.cuh"

struct DeltaChunkArgs {
  const float* rows;           // [T, row_stride]: q of group g at g d, k at k_col + g d, v of head h at v_col + h dv
  long long row_stride;
  int k_col, v_col;
  const float* beta;           // [T, H]
  const float* decay;          // [T, H]
  float* state;                // [slots, H, dv, d]
  float* even;                 // [tiles][H][d][dv]: the state before a tile's first chunk
  float* odd;                  // [tiles][H][d][dv]: and before its second
  float* factor;               // [2 tiles][H]: a chunk's whole decay
  float* w;                    // [2 tiles][H][64][D]
  float* k;                    // [2 tiles][G][D][64]
  float* tail;                 // [2 tiles][H][64]: what a chunk's end leaves of a token's write
  int* bad;                    // [2 tiles][H]: a write of the chunk is no number
  float* o_raw;                // [T, H dv]: V', then U, then the result
  const int* tile_seq;         // tiles of 128 tokens: sequence and first token of its portion; a sequence's side by side in their order
  const int* tile_q0;
  int tiles;
  const int* cu_q_lens;
  const int* context_lens;
  const int* state_slots;
  int B, G, H, d, dv;
  int heads;                   // of one block (they share q and k)
  int* status;
};

enum { DC_ERR_WAIT = 91 };

#define DC_C 64                // tokens of a chunk
#define DC_THREADS 128
#define DC_COLS 16             // value columns of one block of delta_states
#define DC_AP (DC_C + 4)
#define DC_HEADS 4             // most heads of one block: a warp each sums its logarithms
#define DC_STAGES 3
#define DC_SLICE 16            // terms of a slice of delta_rows

// Two float32 multiply-adds, and two additions, in one instruction.
__device__ __forceinline__ void dc_fma2(float2& c, float2 a, float2 b) {
  unsigned long long& d = reinterpret_cast<unsigned long long&>(c);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}
__device__ __forceinline__ void dc_add2(float2& c, float2 a) {
  unsigned long long& d = reinterpret_cast<unsigned long long&>(c);
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(reinterpret_cast<unsigned long long&>(a)));
}
__device__ __forceinline__ float2 dc_mul2(float2 a, float2 b) {
  float2 c;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(c))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return c;
}
// c += the products of four neighbours, even and odd ones apart; the first four of a sum
__device__ __forceinline__ void dc_fma4_first(float2& c, const float4& a, const float4& b) {
  c = dc_mul2(make_float2(a.x, a.y), make_float2(b.x, b.y));
  dc_fma2(c, make_float2(a.z, a.w), make_float2(b.z, b.w));
}
__device__ __forceinline__ void dc_fma4(float2& c, const float4& a, const float4& b) {
  dc_fma2(c, make_float2(a.x, a.y), make_float2(b.x, b.y));
  dc_fma2(c, make_float2(a.z, a.w), make_float2(b.z, b.w));
}

// log2 of a decay; one of 0 (its exponential underflowed) stays finite and still wipes out what came before.  NaN stays NaN.
__device__ __forceinline__ float dc_log2(float g) {
  const float l = log2f(g);
  return l < -2000.f ? -2000.f : l;
}
// By one warp: the running sums of the logarithms of a head's decays over a chunk's n tokens.  Returns their whole sum.
__device__ __forceinline__ double dc_sums(const DeltaChunkArgs& p, int t0, int n, int h, double (&L)[DC_C]) {
  const int lane = threadIdx.x & 31;
  double a[2], s = 0.0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int j = 2 * lane + i;
    s += (double)(j < n ? dc_log2(p.decay[(size_t)(t0 + j) * p.H + h]) : 0.f);
    a[i] = s;
  }
  double incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  double before = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane == 0) before = 0.0;                         // (not incl - s: a NaN would reach the lane's tokens before it)
#pragma unroll
  for (int i = 0; i < 2; ++i) L[2 * lane + i] = before + a[i];
  return __shfl_sync(0xffffffffu, incl, 31);
}
__device__ __forceinline__ float dc_ratio(double a, double b) { return exp2f((float)(a - b)); }

__device__ __forceinline__ void dc_copy(float* to, const float* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(tc_smem(to)), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// x_i . y_j over D values: rows 8 r of x and 16 s of y (pitch D + 4), those with 16 s <= 8 r + 7; sixteen terms a sum.
template <int D> __device__ __forceinline__ void dc_scores(float (&out)[8][4], const float* x, const float* y) {
  constexpr int KP = D + 4;
#pragma unroll 1
  for (int e = 0; e < D; e += 16) {
    float2 acc[8][4];
#pragma unroll
    for (int u = 0; u < 16; u += 4) {
      float4 b[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) b[s] = *reinterpret_cast<const float4*>(y + 16 * s * KP + e + u);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float4 a = *reinterpret_cast<const float4*>(x + 8 * r * KP + e + u);
#pragma unroll
        for (int s = 0; s <= r / 2; ++s) {
          if (u == 0) dc_fma4_first(acc[r][s], a, b[s]);
          else dc_fma4(acc[r][s], a, b[s]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int s = 0; s <= r / 2; ++s) {
        const float sum = acc[r][s].x + acc[r][s].y;
        out[r][s] = e == 0 ? sum : out[r][s] + sum;
      }
  }
}
// By the whole block: the copies of a barrier's phase are there.  If they do not come: false for all, the status set, after as long
// again for what is still on its way.
__device__ __forceinline__ bool dc_arrived(unsigned bar, unsigned parity, int* status) {
  if (__syncthreads_and(mbar_wait(bar, parity))) return true;
  if (threadIdx.x == 0) {
    atomicExch(status, DC_ERR_WAIT);
    mbar_wait(bar, parity);
  }
  __syncthreads();
  return false;
}
// Row t < n of d values to the row of D values of a tile, the rest of it zeros; by one thread a row.
template <int D> __device__ __forceinline__ void dc_fetch_row(float* to, const float* src, bool there, int d, unsigned bar) {
  if (there) dc_copy(to, src, 4 * d, bar);
  for (int c = there ? d : 0; c < D; c += 4) *reinterpret_cast<float4*>(to + c) = make_float4(0.f, 0.f, 0.f, 0.f);
}

// ---------------------------------------------------------------- the triangular systems
// grid (2 tiles, H / heads): a chunk of `heads` heads that share k.  The products k_i . k_j once, in registers; then per head A, and
// the columns of [b G K | b V], two a thread, sixteen tokens at a time: what the blocks of tokens before leave (pairs of terms, sixteen
// a sum), then the block's own substitution.  A value that is no number reaches the tokens behind it only.
// What bounds it: shared memory in the products (a 16-byte read takes 2 clocks of a multiprocessor where eight lanes have at most two
// addresses, else 4: a warp's 18 reads 40 clocks, 8 warps 320, for 256 of multiply-adds; with one column a thread 288 for 128), 22 k of a
// block's 55 k clocks (two heads), then k_i . k_j 8 k.
template <int D>
__global__ void __launch_bounds__(DC_THREADS, 2) delta_solve_kernel(const DeltaChunkArgs p) {
  extern __shared__ __align__(16) float dc_sm[];
  constexpr int KP = D + 4, W = 2 * DC_THREADS;
  float* ks = dc_sm;                                   // [64][KP]
  float* at = ks + DC_C * KP;                          // [i][DC_AP]: A_ij (j < i)
  float4* xs = reinterpret_cast<float4*>(at + DC_C * DC_AP);       // [12][W]: a column's first 48 tokens (a thread reads its own)
  __shared__ double L[DC_HEADS][DC_C];
  __shared__ float bs[DC_HEADS][DC_C], bg[DC_HEADS][DC_C];
  __shared__ __align__(8) unsigned long long bars[1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h0 = blockIdx.y * p.heads, chunk = blockIdx.x;
  const int b = p.tile_seq[chunk >> 1], q0 = p.tile_q0[chunk >> 1] + DC_C * (chunk & 1);
  const int qlen = p.cu_q_lens[b + 1] - p.cu_q_lens[b], t0 = p.cu_q_lens[b] + q0, n = min(DC_C, qlen - q0), rep = p.H / p.G;
  pdl_trigger();
  pdl_wait();
  if (n <= 0) return;
  const unsigned bar = tc_smem(bars);
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(bar, 4 * n * p.d);
  }
  __syncthreads();
  if (tid < DC_C) dc_fetch_row<D>(ks + tid * KP, p.rows + (size_t)(t0 + tid) * p.row_stride + p.k_col + (size_t)(h0 / rep) * p.d, tid < n, p.d, bar);
  if (warp < p.heads) {
    const int h = h0 + warp;
    const double all = dc_sums(p, t0, n, h, L[warp]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = 2 * lane + i;
      const double l = L[warp][j];                     // (this lane's own)
      const float f = j < n ? p.beta[(size_t)(t0 + j) * p.H + h] : 0.f;
      bs[warp][j] = f;
      bg[warp][j] = f * exp2f((float)l);
      p.tail[((size_t)chunk * p.H + h) * DC_C + j] = dc_ratio(all, l);
    }
    if (lane == 0) {
      p.factor[(size_t)chunk * p.H + h] = exp2f((float)all);
      p.bad[(size_t)chunk * p.H + h] = 0;
    }
  }
  if (!dc_arrived(bar, 0, p.status)) return;
  if (h0 % rep == 0) {                                 // K for delta_states: tokens side by side
    float* o = p.k + ((size_t)chunk * p.G + h0 / rep) * DC_C * D;
    for (int e = tid; e < DC_C * (D / 4); e += DC_THREADS) {
      const int t = e % DC_C, c = (e / DC_C) << 2;
      const float4 v = *reinterpret_cast<const float4*>(ks + t * KP + c);
      o[c * DC_C + t] = v.x; o[(c + 1) * DC_C + t] = v.y; o[(c + 2) * DC_C + t] = v.z; o[(c + 3) * DC_C + t] = v.w;
    }
  }
  // k_i . k_j: rows bi + 8 r, columns bj + 16 s, those that reach below the diagonal
  const int bi = tid >> 4, bj = tid & 15;
  float kk[8][4];
  dc_scores<D>(kk, ks + bi * KP, ks + bj * KP);
  const int cols = D + p.dv;
  const size_t upitch = (size_t)p.H * p.dv;
  for (int hh = 0; hh < p.heads; ++hh) {
    const int h = h0 + hh;
    if (hh > 0) __syncthreads();                       // the head before is done with A
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int s = 0; s <= r / 2; ++s) {
        const int i = bi + 8 * r, j = bj + 16 * s;
        if (j < i) at[i * DC_AP + j] = bs[hh][i] * dc_ratio(L[hh][i], L[hh][j]) * kk[r][s];
      }
    __syncthreads();
    float* w = p.w + ((size_t)chunk * p.H + h) * DC_C * D;
    const float* vr = p.rows + (size_t)t0 * p.row_stride + p.v_col + (size_t)h * p.dv;
    float* u = p.o_raw + (size_t)t0 * upitch + (size_t)h * p.dv;
#pragma unroll 1
    for (int c0 = tid; c0 < cols; c0 += W) {
      // of K a column is read from shared memory, of V from the rows, a block of tokens ahead
      const bool key[2] = {c0 < D, c0 + DC_THREADS < D}, there[2] = {true, c0 + DC_THREADS < cols};
      float x[2][16];
      auto ahead = [&](int blk) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
          if (!key[m]) {
            const float* src = vr + (size_t)(16 * blk) * p.row_stride + (c0 + m * DC_THREADS - D);
#pragma unroll
            for (int i = 0; i < 16; ++i, src += p.row_stride) x[m][i] = there[m] && 16 * blk + i < n ? *src : 0.f;
          }
      };
      ahead(0);
#pragma unroll 1
      for (int blk = 0; 16 * blk < n; ++blk) {         // sixteen tokens (past the portion's end nobody reads W)
        float2 acc[2][16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[0][i] = acc[1][i] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int jb = 0; jb < 4 * blk; ++jb) {         // four tokens before them
          const float4 y0 = xs[jb * W + tid], y1 = xs[jb * W + DC_THREADS + tid];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(at + (16 * blk + i) * DC_AP + 4 * jb);
            dc_fma4(acc[0][i], a, y0);
            dc_fma4(acc[1][i], a, y1);
          }
        }
        float y[2][16];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const float* f = key[m] ? bg[hh] : bs[hh];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (key[m]) x[m][i] = ks[(16 * blk + i) * KP + c0 + m * DC_THREADS];
            y[m][i] = f[16 * blk + i] * x[m][i];
          }
        }
        if (16 * (blk + 1) < n) ahead(blk + 1);
        float own[2][16];                              // what the block's own tokens leave
#pragma unroll
        for (int i = 0; i < 16; ++i) own[0][i] = own[1][i] = 0.f;
#pragma unroll
        for (int q = 0; q < 16; q += 4) {              // four tokens: one after the other, then what they leave to those behind them
#pragma unroll
          for (int i = q; i < 16; ++i) {
            const float4 a4 = *reinterpret_cast<const float4*>(at + (16 * blk + i) * DC_AP + 16 * blk + q);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
            for (int m = 0; m < 2; ++m) {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (q + e < i) own[m][i] = fmaf(a[e], y[m][q + e], own[m][i]);
              if (i < q + 4) y[m][i] -= own[m][i] + (acc[m][i].x + acc[m][i].y);
            }
          }
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int c = c0 + m * DC_THREADS;
          if (blk < 3) {
#pragma unroll
            for (int g = 0; g < 4; ++g)
              xs[(4 * blk + g) * W + m * DC_THREADS + tid] = make_float4(y[m][4 * g], y[m][4 * g + 1], y[m][4 * g + 2], y[m][4 * g + 3]);
          }
          if (key[m]) {
            float* o = w + 16 * blk * D + c;
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i * D] = y[m][i];
          } else if (there[m]) {
            float* o = u + (size_t)(16 * blk) * upitch + (c - D);
#pragma unroll
            for (int i = 0; i < 16; ++i, o += upitch)
              if (16 * blk + i < n) *o = y[m][i];
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------- the states, one chunk after the other
// grid (dv / 16, H, B), four warps, two blocks a multiprocessor.  U of a chunk: a warp has sixteen tokens, a lane sixteen (D = 64: eight)
// of d and four columns, its part of S in registers; the eight lanes that share columns add up.  Then S: a warp has a quarter of d, a
// lane sixteen tokens and four columns, U in registers, and the lanes again add up; a value of S belongs to one lane and is carried in
// a register.  Only S and U pass through shared memory, W and K of a chunk are fetched while the other one is worked on.  A lane's 16
// bytes of W or K serve four columns and two lanes of eight read the same ones, 2 clocks of shared memory a read, so that the
// multiply-adds bound it: 2048 clocks of a multiprocessor a chunk and sixteen columns, keys of 128; it takes 4.1 k, two blocks beside
// one another (products 3.1 k, update 3.1 k of a block's 8.3 k: beside the multiply-adds half as many other instructions, and two warps a
// scheduler cannot hide all that each waits for; the rest is S, U and V' to and from memory).
template <int D>
__global__ void __launch_bounds__(DC_THREADS, 2) delta_states_kernel(const DeltaChunkArgs p) {
  extern __shared__ __align__(16) float dc_sm[];
  constexpr int NI = D / 32, SP = D + 8, UP = DC_C + 8, OWN = D / 8, TILE = DC_C * D;
  float* ws = dc_sm;                                   // [64][D]
  float* kt = ws + TILE;                               // [D][64]
  float* ss = kt + TILE;                               // [16 columns][SP]: S, groups of four values of d at places exchanged by column
  float* us = ss + DC_COLS * SP;                       // [16 columns][UP]: what of U reaches the chunk's end, likewise
  float* tails = us + DC_COLS * UP;                    // [64]
  __shared__ __align__(8) unsigned long long bars[2];  // W and tails, K
  __shared__ int first_s;
  const int b = blockIdx.z, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slot = p.state_slots[b], s0 = p.cu_q_lens[b], qlen = p.cu_q_lens[b + 1] - s0, d = p.d;
  const unsigned bar_w = tc_smem(&bars[0]), bar_k = tc_smem(&bars[1]);
  if (tid == 0) {
    first_s = -1;
    mbar_init(bar_w, 1);
    mbar_init(bar_k, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  for (int i = tid; i < p.tiles; i += DC_THREADS)      // the sequence's first tile
    if (p.tile_seq[i] == b && p.tile_q0[i] == 0) first_s = i;
  __syncthreads();
  const int first = first_s;
  if (first < 0) { pdl_trigger(); pdl_wait(); return; }
  const bool carry = slot >= 0 && p.context_lens[b] - qlen > 0;
  const int chunks = (qlen + DC_C - 1) / DC_C, col0 = blockIdx.x * DC_COLS;
  // lanes: cg four columns 4 cg ..; of U dg four values of d of every 32, of S tg four tokens of every 16 and half: of two values of d
  const int cg = lane & 3, dg = lane >> 2, tg = dg & 3, half = lane >> 4;
  const bool b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
  const int cc = (b3 ? 2 : 0) + (b2 ? 1 : 0), mine = 4 * cg + cc;  // the column of which this lane gets sums
  auto s_at = [&](int e) { return (4 * cc + cg) * SP + (((e >> 2) ^ cc) << 2) + (e & 3); };        // of column `mine`
  auto u_at = [&](int t) { return (4 * cc + cg) * UP + (((t >> 2) ^ cc) << 2) + (t & 3); };
  const float* wg = p.w + ((size_t)(2 * first) * p.H + h) * TILE;
  const float* tail_g = p.tail + ((size_t)(2 * first) * p.H + h) * DC_C;
  const float* kg = p.k + ((size_t)(2 * first) * p.G + h / (p.H / p.G)) * TILE;
  auto fetch_w = [&](int c) {                          // by one thread
    mbar_expect_tx(bar_w, 4 * (TILE + DC_C));
    dc_copy(ws, wg + (size_t)c * p.H * TILE, 4 * TILE, bar_w);
    dc_copy(tails, tail_g + (size_t)c * p.H * DC_C, 4 * DC_C, bar_w);
  };
  auto fetch_k = [&](int c) {
    mbar_expect_tx(bar_k, 4 * TILE);
    dc_copy(kt, kg + (size_t)c * p.G * TILE, 4 * TILE, bar_k);
  };
  pdl_wait();
  if (tid == 0) { fetch_w(0); fetch_k(0); }
  float* shead = p.state + ((size_t)max(slot, 0) * p.H + h) * p.dv * d + (size_t)col0 * d;
  for (int e = tid; e < DC_COLS * (D / 4); e += DC_THREADS) {
    const int c = e / (D / 4), q = e % (D / 4);
    const float4 v = carry && 4 * q < d ? *reinterpret_cast<const float4*>(shead + (size_t)c * d + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(ss + (4 * (c & 3) + (c >> 2)) * SP + ((q ^ (c & 3)) << 2)) = v;
  }
  // of U this lane gets tokens 16 warp + 2 x + half, of S d = dl + 2 x
  const int tl = 16 * warp + half, dl = warp * (D / 4) + half;
  const size_t upitch = (size_t)p.H * p.dv;
  float* ur = p.o_raw + (size_t)(s0 + tl) * upitch + (size_t)h * p.dv + col0 + mine;
  float vn[8], fn;
  auto ahead = [&](int c) {                            // V' and the whole decay of chunk c
    const float* v = ur + (size_t)(DC_C * c) * upitch;
#pragma unroll
    for (int x = 0; x < 8; ++x, v += 2 * upitch) vn[x] = DC_C * c + tl + 2 * x < qlen ? *v : 0.f;
    fn = p.factor[(size_t)(2 * first + c) * p.H + h];
  };
  ahead(0);
  __syncthreads();
  float own[OWN];
#pragma unroll
  for (int x = 0; x < OWN; ++x) own[x] = ss[s_at(dl + 2 * x)];
  bool ok = true;
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    if (c > 0 || carry) {                              // the state before the chunk (else nobody reads it)
      float* o = (c & 1 ? p.odd : p.even) + ((size_t)(first + (c >> 1)) * p.H + h) * d * p.dv + col0;
      for (int e = tid; e < 4 * d; e += DC_THREADS) {  // four columns of a value of d
        const int q = e & 3, x = e >> 2;
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = ss[(4 * i + q) * SP + (((x >> 2) ^ i) << 2) + (x & 3)];
        *reinterpret_cast<float4*>(o + (size_t)x * p.dv + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
    {
      float4 s[NI][4];
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[i][e] = *reinterpret_cast<const float4*>(ss + (4 * e + cg) * SP + (((dg + 8 * i) ^ e) << 2));
      ok = mbar_wait(bar_w, c & 1);
      const float* wl = ws + 16 * warp * D + 4 * dg;
      // (all sums first, stored behind the loop: a store or a branch in between would keep the next tokens' products from starting)
#pragma unroll
      for (int x = 0; x < 8; ++x) {                    // two tokens
        float2 acc[2][4];
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const float4 y = *reinterpret_cast<const float4*>(wl + (2 * x + t) * D + 32 * i);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (i == 0) dc_fma4_first(acc[t][e], y, s[i][e]);
              else dc_fma4(acc[t][e], y, s[i][e]);
            }
          }
        // eight sums, one for each of the lanes that share the columns
        float v[4], z[2];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float v0 = acc[0][e].x + acc[0][e].y, v1 = acc[1][e].x + acc[1][e].y;
          v[e] = (b4 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, b4 ? v0 : v1, 16);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) z[e] = (b3 ? v[2 + e] : v[e]) + __shfl_xor_sync(0xffffffffu, b3 ? v[e] : v[2 + e], 8);
        vn[x] -= (b2 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, b2 ? z[0] : z[1], 4);
      }
      bool fine = true;
      float* uo = ur + (size_t)(DC_C * c) * upitch;
#pragma unroll
      for (int x = 0; x < 8; ++x, uo += 2 * upitch) {
        const bool there = DC_C * c + tl + 2 * x < qlen;
        if (there) *uo = vn[x];
        fine = fine && (!there || fabsf(vn[x]) <= 3.402823466e38f);
        us[u_at(tl + 2 * x)] = there ? vn[x] * tails[tl + 2 * x] : 0.f;
      }
      if (!fine) p.bad[(size_t)(2 * first + c) * p.H + h] = 1;
    }
    const float factor = fn;
    ok = mbar_wait(bar_k, c & 1) && ok;
    if (!__syncthreads_and(ok)) {                      // a copy did not come: the state is not written; no copy is left on its way
      if (tid == 0) {
        atomicExch(p.status, DC_ERR_WAIT);
        mbar_wait(bar_w, c & 1);
        mbar_wait(bar_k, c & 1);
      }
      __syncthreads();
      pdl_trigger();
      return;
    }
    if (c + 1 < chunks) {
      if (tid == 0) fetch_w(c + 1);
      ahead(c + 1);
    }
    {
      float4 u[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) u[i][e] = *reinterpret_cast<const float4*>(us + (4 * e + cg) * UP + (((tg + 4 * i) ^ e) << 2));
      const float* kl = kt + dl * DC_C + 4 * tg;
#pragma unroll
      for (int x = 0; x < OWN; ++x) {
        float2 acc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 y = *reinterpret_cast<const float4*>(kl + 2 * x * DC_C + 16 * i);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (i == 0) dc_fma4_first(acc[e], y, u[i][e]);
            else dc_fma4(acc[e], y, u[i][e]);
          }
        }
        float v[4], z[2];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = acc[e].x + acc[e].y;
#pragma unroll
        for (int e = 0; e < 2; ++e) z[e] = (b3 ? v[2 + e] : v[e]) + __shfl_xor_sync(0xffffffffu, b3 ? v[e] : v[2 + e], 8);
        own[x] = fmaf(factor, own[x], (b2 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, b2 ? z[0] : z[1], 4));
      }
#pragma unroll
      for (int x = 0; x < OWN; ++x) ss[s_at(dl + 2 * x)] = own[x];
    }
    __syncthreads();
    if (tid == 0 && c + 1 < chunks) fetch_k(c + 1);
  }
  pdl_trigger();                                       // only now: blocks of the next kernel that wait on a multiprocessor take room there
  if (slot < 0) return;
  for (int e = tid; e < DC_COLS * (D / 4); e += DC_THREADS) {
    const int c = e / (D / 4), q = e % (D / 4);
    if (4 * q < d) *reinterpret_cast<float4*>(shead + (size_t)c * d + 4 * q) = *reinterpret_cast<const float4*>(ss + (4 * (c & 3) + (c >> 2)) * SP + ((q ^ (c & 3)) << 2));
  }
}

// ---------------------------------------------------------------- the rows
// grid (2 tiles, H / heads, columns / (16 CPT)), four warps, two blocks a multiprocessor.  The products q_i . k_j once, in registers;
// per head the weights of the chunk's own tokens, then [q | weights] times [S | U] in slices of sixteen terms, which are copied
// two slices ahead: eight rows (every fourth of 32) and CPT columns a thread, pairs of columns an instruction.  The result takes U's
// place.  Where U holds a value that is no number (rare: delta_states says so) weights of 0 are left out instead of multiplied.
// What bounds it: the multiply-adds, 64 x 128 x (128 + 48) a chunk and head (keys and values of 128): 11.3 k clocks, with two blocks
// beside one another 25 k of a head's 33 k; 256 blocks of two heads are one turn of the machine, but two a multiprocessor on 108 only.
template <int D, int CPT>
__global__ void __launch_bounds__(DC_THREADS, 2) delta_rows_kernel(const DeltaChunkArgs p) {
  extern __shared__ __align__(16) float dc_sm[];
  constexpr int KP = D + 4, COLS = 16 * CPT, SLICE = DC_SLICE * COLS, N2 = CPT / 2;
  float* qs = dc_sm;                                   // [64][KP]
  float* ps = qs + DC_C * KP;                          // [64][DC_AP]: the weights
  float* ring = ps + DC_C * DC_AP;                     // [stages][16][COLS]
  float* ks = ps;                                      // [64][KP], until the products are there
  __shared__ double L[DC_HEADS][DC_C];
  __shared__ __align__(8) unsigned long long bars[DC_STAGES + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h0 = blockIdx.y * p.heads, chunk = blockIdx.x, c0 = blockIdx.z * COLS;
  const int b = p.tile_seq[chunk >> 1], q0 = p.tile_q0[chunk >> 1] + DC_C * (chunk & 1);
  const int qlen = p.cu_q_lens[b + 1] - p.cu_q_lens[b], t0 = p.cu_q_lens[b] + q0, n = min(DC_C, qlen - q0), d = p.d;
  pdl_trigger();
  pdl_wait();
  if (n <= 0) return;
  const float* rq = p.rows + (size_t)t0 * p.row_stride + (size_t)(h0 / (p.H / p.G)) * d;
  const unsigned bar0 = tc_smem(bars), bar_qk = bar0 + 8 * DC_STAGES;
  if (tid == 0) {
    for (int i = 0; i <= DC_STAGES; ++i) mbar_init(bar0 + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(bar_qk, 8 * n * d);
  }
  __syncthreads();
  {
    const int t = tid % DC_C;
    const float* src = rq + (size_t)t * p.row_stride + (tid < DC_C ? 0 : p.k_col);
    dc_fetch_row<D>((tid < DC_C ? qs : ks) + t * KP, src, t < n, d, bar_qk);
  }
  if (warp < p.heads) dc_sums(p, t0, n, h0 + warp, L[warp]);
  if (!dc_arrived(bar_qk, 0, p.status)) return;
  // q_i . k_j: rows ty + 8 r, columns tx + 16 s, those that reach the diagonal or below
  const int ty = tid >> 4, tx = tid & 15;
  float sc[8][4];
  dc_scores<D>(sc, qs + ty * KP, ks + tx * KP);
  const bool state = q0 > 0 || (p.state_slots[b] >= 0 && p.context_lens[b] - qlen > 0);
  const int nd = state ? d / DC_SLICE : 0, slices = nd + (n + DC_SLICE - 1) / DC_SLICE;
  const size_t upitch = (size_t)p.H * p.dv;
  const int width = min(COLS, p.dv - c0);
  const int row0 = 32 * (warp >> 1) + (lane >> 3), cx = 4 * ((lane & 7) + 8 * (warp & 1));       // rows row0 + 4 r; columns cx .., 64 + cx ..
  for (int hh = 0; hh < p.heads; ++hh) {
    const int h = h0 + hh;
    const float* sg = (chunk & 1 ? p.odd : p.even) + ((size_t)(chunk >> 1) * p.H + h) * d * p.dv + c0;
    float* ug = p.o_raw + (size_t)t0 * upitch + (size_t)h * p.dv + c0;
    const bool bad = p.bad[(size_t)chunk * p.H + h] != 0;
    // A slice of S is one piece where its rows have COLS columns; else rows are copied one by one, four a warp (a copy is some 60
    // clocks of the thread that asks for it: with all sixteen in one warp the block waited a third of its time)
    auto fetch = [&](int s) {
      if (s >= slices) return;
      const int stage = (hh * slices + s) % DC_STAGES, j = DC_SLICE * (s - nd), rows = s < nd ? DC_SLICE : min(DC_SLICE, n - j), r = 4 * warp + lane;
      const unsigned bar = bar0 + 8 * stage;
      float* to = ring + stage * SLICE;
      if (tid == 0) mbar_expect_tx(bar, 4 * rows * width);
      if (s < nd && p.dv == COLS) {
        if (tid == 0) dc_copy(to, sg + (size_t)(DC_SLICE * s) * COLS, 4 * SLICE, bar);
      } else if (lane < 4 && r < rows) {
        dc_copy(to + r * COLS, s < nd ? sg + (size_t)(DC_SLICE * s + r) * p.dv : ug + (size_t)(j + r) * upitch, 4 * width, bar);
      }
    };
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();                                   // the keys, or the head before's weights and slices, are done with
    fetch(0);
    fetch(1);
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int i = ty + 8 * r, j = tx + 16 * s;
        if (s > r / 2) ps[i * DC_AP + j] = 0.f;
        else ps[i * DC_AP + j] = j <= i ? sc[r][s] * dc_ratio(L[hh][i], L[hh][j]) : 0.f;
      }
    float2 sum[8][N2];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int e = 0; e < N2; ++e) sum[r][e] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int s = 0; s < slices; ++s) {
      const int q = hh * slices + s;
      if (!__syncthreads_and(mbar_wait(bar0 + 8 * (q % DC_STAGES), q / DC_STAGES & 1))) {        // it did not come: nothing is left on its way
        if (tid == 0) {
          atomicExch(p.status, DC_ERR_WAIT);
          mbar_wait(bar0 + 8 * (q % DC_STAGES), q / DC_STAGES & 1);
          if (s + 1 < slices) mbar_wait(bar0 + 8 * ((q + 1) % DC_STAGES), (q + 1) / DC_STAGES & 1);
        }
        __syncthreads();
        return;
      }
      fetch(s + 2);
      if (s == nd) {                                   // the state's part is there: its decay
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float g = exp2f((float)L[hh][row0 + 4 * r]);
#pragma unroll
          for (int e = 0; e < N2; ++e) { sum[r][e].x *= g; sum[r][e].y *= g; }
        }
      }
      const int j0 = DC_SLICE * (s - nd);              // the slice's first token, where it is of U
      if (j0 > 32 * (warp >> 1) + 31) continue;        // behind all of this warp's rows
      const float* a0 = s < nd ? qs + row0 * KP + DC_SLICE * s : ps + row0 * DC_AP + j0;
      const int pitch = 4 * (s < nd ? KP : DC_AP);
      const float* b0 = ring + q % DC_STAGES * SLICE + cx;
      float2 part[8][N2];
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int e = 0; e < N2; ++e) part[r][e] = make_float2(0.f, 0.f);
      if (s >= nd && (bad || j0 + DC_SLICE > n)) {     // (past the portion's end the slice holds what was there before)
#pragma unroll 1
        for (int k = 0; k < DC_SLICE; ++k) {
          float2 y[N2];
#pragma unroll
          for (int e = 0; e < N2; ++e) y[e] = *reinterpret_cast<const float2*>(b0 + k * COLS + (e >= 2 ? 60 : 0) + 2 * e);
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const float a = a0[r * pitch + k];
#pragma unroll
            for (int e = 0; e < N2; ++e)
              if (j0 + k <= row0 + 4 * r) dc_fma2(part[r][e], make_float2(a, a), y[e]);
          }
        }
      } else {
#pragma unroll
        for (int u = 0; u < DC_SLICE; u += 4) {
          float4 a[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) a[r] = *reinterpret_cast<const float4*>(a0 + r * pitch + u);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float4 y[CPT / 4];
#pragma unroll
            for (int e = 0; e < CPT / 4; ++e) y[e] = *reinterpret_cast<const float4*>(b0 + (u + k) * COLS + 64 * e);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const float f = k == 0 ? a[r].x : k == 1 ? a[r].y : k == 2 ? a[r].z : a[r].w;
#pragma unroll
              for (int e = 0; e < CPT / 4; ++e) {
                dc_fma2(part[r][2 * e], make_float2(f, f), make_float2(y[e].x, y[e].y));
                dc_fma2(part[r][2 * e + 1], make_float2(f, f), make_float2(y[e].z, y[e].w));
              }
            }
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int e = 0; e < N2; ++e) dc_add2(sum[r][e], part[r][e]);
    }
    // (every slice of U was in shared memory before the last one was begun)
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int e = 0; e < CPT / 4; ++e) {
        const int i = row0 + 4 * r, c = cx + 64 * e;
        if (i < n && c0 + c < p.dv)
          *reinterpret_cast<float4*>(ug + (size_t)i * upitch + c) = make_float4(sum[r][2 * e].x, sum[r][2 * e].y, sum[r][2 * e + 1].x, sum[r][2 * e + 1].y);
      }
  }
}

// ---------------------------------------------------------------- launcher
template <typename K> static int dc_room(K kernel, size_t bytes) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  return e == cudaSuccess ? GG_OK : gg_fail(GG_ERR_CUDA, "delta_chunks: %s", cudaGetErrorString(e));
}
// As many heads of a group a block as leave `blocks` blocks: they share the products of their keys.
static int dc_heads(const DeltaChunkArgs& p, long long blocks) {
  int heads = 1;
  while (heads < DC_HEADS && p.H / p.G % (2 * heads) == 0 && 2ll * p.tiles * (p.H / (2 * heads)) >= blocks) heads *= 2;
  return heads;
}

template <int D, int CPT> static int dc_rows(DeltaChunkArgs p, cudaStream_t stream) {
  constexpr int KP = D + 4, COLS = 16 * CPT, own = DC_C * DC_AP + DC_STAGES * DC_SLICE * COLS;
  const size_t smem = (DC_C * KP + (own > DC_C * KP ? own : DC_C * KP)) * sizeof(float);
  if (const int rc = dc_room(delta_rows_kernel<D, CPT>, smem)) return rc;
  p.heads = dc_heads(p, 222);
  gg_launch(delta_rows_kernel<D, CPT>, dim3(2 * p.tiles, p.H / p.heads, (p.dv + COLS - 1) / COLS), dim3(DC_THREADS), smem, stream, p);
  return gg_check_launch("delta_rows");
}

template <int D> static int dc_run(DeltaChunkArgs p, cudaStream_t stream) {
  const size_t solve = (DC_C * (D + 4) + DC_C * DC_AP + 48 * 2 * DC_THREADS) * sizeof(float);
  if (const int rc = dc_room(delta_solve_kernel<D>, solve)) return rc;
  p.heads = dc_heads(p, 222);
  gg_launch(delta_solve_kernel<D>, dim3(2 * p.tiles, p.H / p.heads), dim3(DC_THREADS), solve, stream, p);
  if (const int rc = gg_check_launch("delta_solve")) return rc;
  const size_t states = (2 * DC_C * D + DC_COLS * (D + 8) + DC_COLS * (DC_C + 8) + DC_C) * sizeof(float);
  if (const int rc = dc_room(delta_states_kernel<D>, states)) return rc;
  gg_launch_after(delta_states_kernel<D>, dim3(p.dv / DC_COLS, p.H, p.B), dim3(DC_THREADS), states, stream, p);
  if (const int rc = gg_check_launch("delta_states")) return rc;
  return p.dv <= 64 ? dc_rows<D, 4>(p, stream) : dc_rows<D, 8>(p, stream);
}

// gg_delta_recur (a decay per head) over the sequences whose chunks of 128 tokens are the tiles (all chunks of a sequence, in their
// order); the others are left alone.  Returns GG_ERR_UNSUPPORTED, and launches nothing, where sizes or addresses are not for
// these kernels.  Scratch the caller provides: float[num_tiles * H * (d * dv + 4)] and float[num_tiles * (128 * (H + G) * D +
// H * (d * dv + 130))] with D = 64 or 128, the first that holds d.
extern "C" int gg_delta_chunks(const float* qkv, const float* beta, const float* decay, float* state, float* scratch,
                               long long scratch_floats, float* w, long long w_floats, const int* tile_seq, const int* tile_q0,
                               int num_tiles, const int* cu_q_lens, const int* context_lens, const int* state_slots, int T, int B,
                               int G, int H, int d, int dv, float* o_raw, int* status, cudaStream_t stream) {
  GG_REQUIRE(T >= 0 && B > 0 && G > 0 && H > 0 && H % G == 0 && d > 0 && dv > 0 && num_tiles >= 0, "delta_chunks: bad sizes T=%d B=%d G=%d H=%d d=%d dv=%d", T, B, G, H, d, dv);
  GG_REQUIRE(qkv && beta && decay && state && scratch && w && o_raw && status, "delta_chunks: a pointer is null");
  const size_t addresses = (size_t)qkv | (size_t)state | (size_t)scratch | (size_t)w | (size_t)o_raw;
  if (d > 128 || d % 32 || dv % DC_COLS || dv > 256 || H > 65535 || B > 65535 || addresses % 16) return GG_ERR_UNSUPPORTED;
  const long long D = d <= 64 ? 64 : 128, tiles = num_tiles, per = (long long)H * d * dv;
  GG_REQUIRE(scratch_floats >= tiles * (per + 4 * H) && w_floats >= tiles * (128 * (H + G) * D + per + 130 * H),
             "delta_chunks: scratch of %lld and %lld values is too small", scratch_floats, w_floats);
  if (num_tiles == 0) return GG_OK;
  DeltaChunkArgs p = {};
  p.rows = qkv; p.row_stride = 2ll * G * d + (long long)H * dv; p.k_col = G * d; p.v_col = 2 * G * d;
  p.beta = beta; p.decay = decay; p.state = state; p.o_raw = o_raw;
  p.even = scratch; p.factor = scratch + tiles * per;
  p.w = w; p.k = p.w + tiles * 128 * H * D; p.odd = p.k + tiles * 128 * G * D; p.tail = p.odd + tiles * per;
  p.bad = reinterpret_cast<int*>(p.tail + tiles * 128 * H);
  p.tile_seq = tile_seq; p.tile_q0 = tile_q0; p.tiles = num_tiles; p.cu_q_lens = cu_q_lens; p.context_lens = context_lens;
  p.state_slots = state_slots; p.B = B; p.G = G; p.H = H; p.d = d; p.dv = dv; p.status = status;
  return d <= 64 ? dc_run<64>(p, stream) : dc_run<128>(p, stream);
}
