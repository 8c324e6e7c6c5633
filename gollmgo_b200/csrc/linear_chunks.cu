// The plain linear recurrence over prompt portions in chunks of 128 tokens, as matrix products on tcgen05.  Per head a state
// S [d, dv]:
//     S <- g_t S + k_t (b_t v_t)^T;    o_t = S^T q_t
// with a decay g and a factor b per token and head (a state-space layer: k = B, q = C, v = x, b = the step size; the matrix
// memory), or one fixed decay a head and b = 1 (retention).  With L_i the sum of log2 g over a chunk's tokens up to i:
//   linear_products  all chunks at once: what a chunk adds to the state, P = sum_j 2^(L_n - L_j) b_j k_j v_j^T, and 2^(L_n);
//                    heads that share k stand side by side in one product
//   linear_scan      element by element, a sequence's chunks one after the other: S' = 2^(L_n) S + P; leaves S before every
//                    chunk where P was
//   linear_rows      all chunks at once: o_i = 2^(L_i) S^T q_i + sum_(j<=i) 2^(L_i - L_j) b_j (q_i . k_j) v_j; heads that share q
//                    and k share the products q_i . k_j.  Retention: then the unit norm and the gate.
// The products are float32 products made of three tf32 ones: x = hi + lo, hi to 11 bits, lo what is left (its first 11
// bits count); hi hi + hi lo + lo hi, the term left out and what lo drops are 2^-21 of a product.  hi hi and the small terms
// have accumulators of their own where tensor memory has the room (the tensor core's sums are cut off, not rounded).  Sums
// of logarithms are formed in float64, so strong decays cost no accuracy.
// Infinities and NaN reach what they reach token by token: a bad value column, factor or decay the rows from its token on, a
// bad k those rows in all columns, a bad q its own row, and the state.  There they are NaN, also where the walk would have
// kept an infinity.  What rounds to infinity at 11 bits (from 2^128 (1 - 2^-12) on; no bfloat16 value does) counts as one.
// What bounds it: reading rows, splitting and writing both parts to shared memory (every operand arrives as float32 rows and
// three of them have to be turned), a step of 32 values of k at a time, the next step's reads under way; the products run
// beside that.  With the products on mma.sync (tf32 there runs at 486 multiply-adds a clock and multiprocessor) every warp
// had to split its fragments again: 215 us for the state-space layer below and 225 for retention.
// Measured (B200), us for the three kernels, before: 2048 tokens of one sequence, a state-space layer of 64 heads of 64 with a
// state of 128: 41 + 9 + 83, token by token 359; 2011 tokens of three, retention of 16 heads 128 x 256: 42 + 9 + 77, packed
// float32 232 (each kernel alone).  Slower: reads two steps ahead (registers spill: rows 130 and 117, where they took 97); groups of four warps with a step each
// (rows 112); two issuers (no change).
// All waits on barriers are bounded; one that runs out sets *status and the CTA winds down.
#include "tc_common.cuh"

#define LC_C 128               // tokens of a chunk
#define LC_THREADS 544         // sixteen warps that read, split and write (with eight everything took half as long again: too few
                               // to wait behind); one that issues the products
#define LC_WORKERS 512
#define LC_ISSUER 16
#define LC_A_BYTES (128 * 128) // a part (hi or lo) of A's tile: 128 rows of 32 tf32 values, 128-byte swizzle

enum { LC_ERR_EMPTY = 81, LC_ERR_FULL = 82, LC_ERR_DONE = 83 };

struct LinearArgs {
  const float* rows;           // [T, row_stride]: q of group g at q_col + g d, k at k_col + g d
  long long row_stride;
  int q_col, k_col;
  const float* values;         // [T, values_stride]: v of head h at h dv
  long long values_stride;
  const float* beta;           // [T, H]; null: 1
  const float* decay;          // [T, H]; null: log2_decay
  const float* log2_decay;     // [H]
  float* state;                // [slots, H, dv, d]
  float* scratch;              // [chunks][H][dv][d]: P of a chunk, then the state before it
  float* factor;               // [chunks][H]: 2^(L_n)
  const int* tile_seq;         // chunks: sequence and first token of its portion; a sequence's side by side in their order
  const int* tile_q0;
  int tiles;
  const int* cu_q_lens;
  const int* context_lens;
  const int* state_slots;
  int B, G, H, d, dv, heads;   // heads: of one CTA (they share a group)
  float* o_raw;                // [T, H dv]
  const void* gate;            // retention: [T, gate_stride]
  long long gate_stride;
  float eps;
  void* out;                   // retention: [T, H dv] in the gate's type
  int* status;
};

// log2 of a decay.  One of 0 (its exponential underflowed) stays finite, so that differences of sums do, and still
// wipes out what came before: 2^-2000.  NaN stays NaN.
__device__ __forceinline__ float lc_log2(float g) {
  const float l = log2f(g);
  return l < -2000.f ? -2000.f : l;
}

// What a lane of a warp holds of a chunk's decays and factors: of tokens 4 lane .. 4 lane + 3.
struct LcTokens { float g[4], b[4]; };
__device__ __forceinline__ LcTokens lc_tokens(const LinearArgs& p, int t0, int n, int h) {
  LcTokens x;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = 4 * (threadIdx.x & 31) + i;
    x.g[i] = j < n && p.decay ? p.decay[(size_t)(t0 + j) * p.H + h] : 1.f;
    x.b[i] = j < n ? (p.beta ? p.beta[(size_t)(t0 + j) * p.H + h] : 1.f) : 0.f;
  }
  return x;
}
// Sums of logarithms as two float32 parts (48 bits).
struct LcSums { float hi[LC_C], lo[LC_C]; };
// By one warp: L (inclusive sums of log2 of the decays) and the factors b [128] of the chunk's n tokens.  Returns their whole sum.
__device__ __forceinline__ double lc_sums(const LinearArgs& p, const LcTokens& x, int n, int h, LcSums& L, float* b) {
  const int lane = threadIdx.x & 31;
  const float fixed = p.decay ? 0.f : p.log2_decay[h];
  double a[4], s = 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = 4 * lane + i;
    s += (double)(j < n ? (p.decay ? lc_log2(x.g[i]) : fixed) : 0.f);
    a[i] = s;
    b[j] = x.b[i];
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
  for (int i = 0; i < 4; ++i) {
    const double l = before + a[i];
    L.hi[4 * lane + i] = (float)l;
    L.lo[4 * lane + i] = (float)(l - (double)(float)l);
  }
  return __shfl_sync(0xffffffffu, before + a[3], 31);
}
// Two to the difference of two such sums, rounded once, as a float64 difference would be: what rounding takes from hi - hi2 goes with the
// small parts.  (Without that, two roundings: a power of 2^-8 to 2^-14 is off by 3.0e-7 instead of 2.0e-7.  With float64 subtractions the
// conversions take longer than these seven instructions: rows of 2048 tokens and 64 heads 97 us against 87.)
__device__ __forceinline__ float lc_power(float hi, float lo, float hi2, float lo2) {
  const float s = hi - hi2, t = s - hi;
  return exp2f(s + (((hi - (s - t)) - (hi2 + t)) + (lo - lo2)));
}

__device__ __forceinline__ void lc_split(float x, float& hi, float& lo) {
  hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
  lo = x - hi;
}
__device__ __forceinline__ void lc_sts4(unsigned addr, float a, float b, float c, float d) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void lc_sts(unsigned addr, float a) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(a) : "memory"); }

// A tile of R rows of 32 values of k, its hi part at `at` and its lo part `lo_off` further.
//   along: row r is 32 neighbouring values in memory.  A thread has the 16-byte piece tid % 8 of rows tid / 8 + 64 i.
//   across: a value of k is a row in memory (a token), r runs along it.  A lane has token `lane`, and eight neighbouring r a
//           turn: r = 8 (warp + 16 i).
template <int R> struct LcAlong {
  static constexpr int N = (R + 63) / 64;
  float4 v[N];
  __device__ __forceinline__ void load(const float* src, long long pitch, int rows, int k0, int kmax) {
    const int c = k0 + ((threadIdx.x & 7) << 2);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int r = (threadIdx.x >> 3) + 64 * i;
      v[i] = r < rows && c < kmax ? *reinterpret_cast<const float4*>(src + (size_t)r * pitch + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  // scale(r): the row's factor
  template <typename F> __device__ __forceinline__ void store(unsigned at, unsigned lo_off, F scale) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int r = (threadIdx.x >> 3) + 64 * i, c = threadIdx.x & 7;
      {
        const float f = scale(r);
        float h[4], l[4];
        lc_split(v[i].x * f, h[0], l[0]); lc_split(v[i].y * f, h[1], l[1]);
        lc_split(v[i].z * f, h[2], l[2]); lc_split(v[i].w * f, h[3], l[3]);
        const unsigned to = at + r * 128 + ((c ^ (r & 7)) << 4);
        lc_sts4(to, h[0], h[1], h[2], h[3]);
        lc_sts4(to + lo_off, l[0], l[1], l[2], l[3]);
      }
    }
  }
};
template <int R> struct LcAcross {
  static constexpr int N = (R + 127) / 128;
  float4 v[2 * N];
  // src: value 0 of token 0 of the step; tokens: how many of the 32 there are; rows: how many values
  __device__ __forceinline__ void load(const float* src, long long pitch, int tokens, int rows) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* s = src + (size_t)(lane < tokens ? lane : 0) * pitch;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = 8 * (warp + 16 * i) + 4 * e;
        v[2 * i + e] = lane < tokens && r < rows ? *reinterpret_cast<const float4*>(s + r) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
  }
  // A product over tokens gives an earlier token's row a weight of 0 for a later one's value, and 0 times infinity or NaN is
  // NaN: after the store such values leave the tile (as 0), and first[r] becomes the first token that had one in column r.  One
  // multiply-add a value finds them.  Returns whether there was any.
  __device__ __forceinline__ bool take_out(unsigned at, unsigned lo_off, int token, int* first) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float z = 0.f;
#pragma unroll
    for (int i = 0; i < 2 * N; ++i) { z = fmaf(v[i].x, 0.f, z); z = fmaf(v[i].y, 0.f, z); z = fmaf(v[i].z, 0.f, z); z = fmaf(v[i].w, 0.f, z); }
    if (z == 0.f) return false;
#pragma unroll
    for (int i = 0; i < 2 * N; ++i) {
      auto check = [&](float x, int e) {
        const int r = 8 * (warp + 16 * (i >> 1)) + e;
        if (x * 0.f == 0.f) return;
        atomicMin(first + r, token);
        const unsigned to = at + r * 128 + (((lane >> 2) ^ e) << 4) + ((lane & 3) << 2);
        lc_sts(to, 0.f);
        lc_sts(to + lo_off, 0.f);
      };
      const int e = 4 * (i & 1);
      check(v[i].x, e); check(v[i].y, e + 1); check(v[i].z, e + 2); check(v[i].w, e + 3);
    }
    return true;
  }
  // scale(i): the factor of the lane's token in the rows of turn i
  template <typename F> __device__ __forceinline__ void store(unsigned at, unsigned lo_off, F scale) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int r0 = 8 * (warp + 16 * i);
      if (R % 128 != 0 && r0 >= R) continue;
      const float f = scale(i);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 q = v[2 * i + (e >> 2)];
        const float x = ((e & 3) == 0 ? q.x : (e & 3) == 1 ? q.y : (e & 3) == 2 ? q.z : q.w) * f;
        float h, l;
        lc_split(x, h, l);
        const unsigned to = at + (r0 + e) * 128 + (((lane >> 2) ^ e) << 4) + ((lane & 3) << 2);      // (r0 + e) % 8 = e
        lc_sts(to, h);
        lc_sts(to + lo_off, l);
      }
    }
  }
};

// D[tmem] (+)= A B, 128 x N x 8 tf32
__device__ __forceinline__ void lc_mma(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc, unsigned idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((unsigned)accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ unsigned lc_idesc(int n) {      // float32 sums, tf32 x tf32, both K-major, M = 128
  return (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(n >> 3) << 17) | ((128u >> 4) << 24);
}
// One step: 32 values of k of a tile pair.  main gets hi hi; small the other two (main too where there is no small).
__device__ __forceinline__ void lc_step(unsigned main, unsigned small, unsigned a, unsigned b, unsigned b_lo, unsigned idesc, bool fresh) {
  const unsigned long long ah = tc_smem_desc(a), al = tc_smem_desc(a + LC_A_BYTES), bh = tc_smem_desc(b), bl = tc_smem_desc(b + b_lo);
  const bool own = small != main;
#pragma unroll
  for (int k = 0; k < 4; ++k) lc_mma(small, al + 2 * k, bh + 2 * k, idesc, !fresh || k > 0);
#pragma unroll
  for (int k = 0; k < 4; ++k) lc_mma(small, ah + 2 * k, bl + 2 * k, idesc, true);
#pragma unroll
  for (int k = 0; k < 4; ++k) lc_mma(main, ah + 2 * k, bh + 2 * k, idesc, !own || !fresh || k > 0);
}

// The ring of stages between the workers and the issuer, as each side sees it.
template <int STAGES> struct LcRing {
  unsigned full0, empty0;
  int s = 0;
  bool ok = true;
  __device__ __forceinline__ int slot() const { return s % STAGES; }
  __device__ __forceinline__ unsigned phase() const { return (s / STAGES) & 1; }
  // worker: the slot may be written
  __device__ __forceinline__ bool wait_empty(const LinearArgs& p, int* abort_s) {
    ok = ok && mbar_wait(empty0 + 8 * slot(), phase() ^ 1);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && (threadIdx.x & 31) == 0) { atomicExch(p.status, LC_ERR_EMPTY); atomicExch(abort_s, 1); }
    return ok;
  }
  // worker: the warp's part of the slot is written
  __device__ __forceinline__ void give() {
    fence_async_smem();
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(full0 + 8 * slot());
    ++s;
  }
  // issuer
  __device__ __forceinline__ bool wait_full(const LinearArgs& p, int* abort_s) {
    ok = ok && mbar_wait(full0 + 8 * slot(), phase());
    if (!ok) { atomicExch(p.status, LC_ERR_FULL); atomicExch(abort_s, 1); }
    tc_fence_after();
    return ok;
  }
  __device__ __forceinline__ void used() { tc_commit(empty0 + 8 * slot()); ++s; }
};

__device__ __forceinline__ bool lc_wait_done(unsigned bar, unsigned parity, const LinearArgs& p, int* abort_s) {
  bool ok = mbar_wait(bar, parity) && !*(volatile int*)abort_s;
  ok = __all_sync(0xffffffffu, ok);
  if (!ok && (threadIdx.x & 31) == 0) { atomicExch(p.status, LC_ERR_DONE); atomicExch(abort_s, 1); }
  tc_fence_after();
  return ok;
}

// ---------------------------------------------------------------- what a chunk adds to the state
// grid (chunks, H / heads, ceil(d / 128)): D [d, heads x dv] over the chunk's tokens.  NB: room for heads x dv columns.
template <int NB>
__global__ void __launch_bounds__(LC_THREADS, 1)
linear_products_kernel(const LinearArgs p) {
  constexpr unsigned B_PART = NB * 128, STAGE = 2 * LC_A_BYTES + 2 * B_PART;
  constexpr int STAGES = 2;
  extern __shared__ unsigned char lc_smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * STAGES + 1];
  __shared__ LcSums Ls[8];
  __shared__ float ws[8][LC_C];
  __shared__ unsigned tmem_base_s;
  __shared__ int abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned base = (tc_smem(lc_smem_raw) + 1023u) & ~1023u;
  const unsigned full0 = tc_smem(&bars[0]), empty0 = tc_smem(&bars[STAGES]), done = tc_smem(&bars[2 * STAGES]);
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 16); mbar_init(empty0 + 8 * s, 1); }
    mbar_init(done, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == LC_ISSUER) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    pdl_trigger();                                     // (not before: a kernel behind could take the tensor memory and wait for this one)
  }
  const int b = p.tile_seq[blockIdx.x], q0 = p.tile_q0[blockIdx.x], h0 = blockIdx.y * p.heads, m0 = blockIdx.z * 128;
  const int qlen = p.cu_q_lens[b + 1] - p.cu_q_lens[b], t0 = p.cu_q_lens[b] + q0, n = min(LC_C, qlen - q0);
  const int d = p.d, dv = p.dv, cols = p.heads * dv, steps = (n + 31) / 32;
  const size_t place = blockIdx.x;
  pdl_wait();
  // the first step's rows and the decays are on their way together
  const float* kb = p.rows + (size_t)t0 * p.row_stride + p.k_col + (size_t)(h0 / (p.H / p.G)) * d + m0;
  const float* vb = p.values + (size_t)t0 * p.values_stride + (size_t)h0 * dv;
  LcAcross<128> a;
  LcAcross<NB> v;
  if (warp < LC_ISSUER) {
    a.load(kb, p.row_stride, n, d - m0);
    v.load(vb, p.values_stride, n, cols);
  }
  if (warp < p.heads) {                                // (at most eight heads)
    const double all = lc_sums(p, lc_tokens(p, t0, n, h0 + warp), n, h0 + warp, Ls[warp], ws[warp]);
    __syncwarp();
    const float hi = (float)all, lo = (float)(all - (double)hi);
#pragma unroll
    for (int i = 0; i < 4; ++i) ws[warp][4 * lane + i] *= lc_power(hi, lo, Ls[warp].hi[4 * lane + i], Ls[warp].lo[4 * lane + i]);
    if (lane == 0 && m0 == 0) p.factor[place * p.H + h0 + warp] = exp2f(hi);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_base_s;
  const int N = (cols + 15) / 16 * 16;
  const unsigned small = NB + N <= 512 ? tmem + NB : tmem;
  LcRing<STAGES> ring{full0, empty0};
  if (warp < LC_ISSUER) {
    const float* wv[LcAcross<NB>::N];                  // the weights of the heads this warp's columns are of
#pragma unroll
    for (int i = 0; i < LcAcross<NB>::N; ++i) wv[i] = ws[min(8 * (warp + 16 * i) / dv, p.heads - 1)] + lane;
    for (int s = 0; s < steps; ++s) {
      if (!ring.wait_empty(p, &abort_s)) break;
      const unsigned at = base + ring.slot() * STAGE;
      a.store(at, LC_A_BYTES, [](int) { return 1.f; });
      v.store(at + 2 * LC_A_BYTES, B_PART, [&](int i) { return wv[i][32 * s]; });
      if (s + 1 < steps) {
        a.load(kb + (size_t)(32 * (s + 1)) * p.row_stride, p.row_stride, n - 32 * (s + 1), d - m0);
        v.load(vb + (size_t)(32 * (s + 1)) * p.values_stride, p.values_stride, n - 32 * (s + 1), cols);
      }
      ring.give();
    }
    if (lc_wait_done(done, 0, p, &abort_s)) {
      // lane = row of the state (of d), so a column of the state is neighbouring lanes
      const int row = m0 + (warp & 3) * 32 + lane;
      const unsigned tl = tmem + ((unsigned)((warp & 3) * 32) << 16), ts = small + ((unsigned)((warp & 3) * 32) << 16);
      for (int c0 = (warp >> 2) * 32; c0 < cols; c0 += 128) {
        unsigned m[32], s[32];
        tc_load32(tl + c0, m);
        if (small != tmem) tc_load32(ts + c0, s);
        if (row < d) {
          float* o = p.scratch + ((place * p.H + h0) * dv + c0) * d + row;
#pragma unroll
          for (int i = 0; i < 32; ++i, o += d) {
            if (c0 + i < cols) *o = __uint_as_float(m[i]) + (small != tmem ? __uint_as_float(s[i]) : 0.f);
          }
        }
      }
    }
  } else if (lane == 0) {
    const unsigned idesc = lc_idesc(N);
    for (int s = 0; s < steps; ++s) {
      if (!ring.wait_full(p, &abort_s)) break;
      const unsigned at = base + ring.slot() * STAGE;
      lc_step(tmem, small, at, at + 2 * LC_A_BYTES, B_PART, idesc, s == 0);
      ring.used();
    }
    tc_commit(done);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == LC_ISSUER) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---------------------------------------------------------------- the state before every chunk
// grid (B, H, pieces of 1024 values), 256 threads, four values a thread; four chunks' reads under way.
__global__ void __launch_bounds__(256)
linear_scan_kernel(const LinearArgs p) {
  __shared__ int first_s;
  pdl_trigger();
  const int b = blockIdx.x, h = blockIdx.y;
  const int slot = p.state_slots[b], qlen = p.cu_q_lens[b + 1] - p.cu_q_lens[b];
  if (threadIdx.x == 0) first_s = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < p.tiles; i += 256)                    // the sequence's first chunk
    if (p.tile_seq[i] == b && p.tile_q0[i] == 0) first_s = i;
  __syncthreads();
  const int first = first_s;
  if (slot < 0 || first < 0) { pdl_wait(); return; }                  // sequences without chunks go through another kernel
  const size_t size = (size_t)p.d * p.dv, at = ((size_t)blockIdx.z * 256 + threadIdx.x) << 2;
  const bool live = at < size;
  float4* st = reinterpret_cast<float4*>(p.state + ((size_t)slot * p.H + h) * size + at);
  pdl_wait();
  if (!live) return;
  const bool carry = p.context_lens[b] - qlen > 0;
  float4 S = carry ? *st : make_float4(0.f, 0.f, 0.f, 0.f);
  const int chunks = (qlen + LC_C - 1) / LC_C;
  auto place = [&](int c) { return (size_t)(first + c) * p.H + h; };
  for (int c0 = 0; c0 < chunks; c0 += 4) {
    float4 P[4];
    float f[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u < chunks) {
        P[u] = *reinterpret_cast<const float4*>(p.scratch + place(c0 + u) * size + at);
        f[u] = p.factor[place(c0 + u)];
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u < chunks) {
        if (c0 + u > 0 || carry) *reinterpret_cast<float4*>(p.scratch + place(c0 + u) * size + at) = S;      // (else nobody reads it)
        S = make_float4(fmaf(f[u], S.x, P[u].x), fmaf(f[u], S.y, P[u].y), fmaf(f[u], S.z, P[u].z), fmaf(f[u], S.w, P[u].w));
      }
  }
  *st = S;
}

// ---------------------------------------------------------------- the rows of every chunk
// grid (chunks, H / heads).  Tensor memory: scores [0, 128), their small terms [128, 256), then O of a head: two buffers of
// main and small for up to 64 columns, one of both for up to 128, main alone for up to 256.
template <int NB, bool RETENTION, typename TA>
__global__ void __launch_bounds__(LC_THREADS, 1)
linear_rows_kernel(const LinearArgs p) {
  constexpr int BR = NB > 128 ? NB : 128;              // rows of a stage's B tile: 128 keys, or the head's columns
  constexpr unsigned B_PART = BR * 128, STAGE = 2 * LC_A_BYTES + 2 * B_PART;
  constexpr int STAGES = NB > 128 ? 2 : 3;
  constexpr int BUFS = NB <= 64 ? 2 : 1;
  extern __shared__ unsigned char lc_smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * STAGES + 3];
  __shared__ __align__(16) LcSums Ls[8];
  __shared__ __align__(16) float bs[8][LC_C];
  __shared__ float fs[8][LC_C];
  __shared__ int first_s[8][NB], marked_s[8];          // of the heads' columns: the first token with infinity or NaN in v
  __shared__ unsigned tmem_base_s;
  __shared__ int abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned base = (tc_smem(lc_smem_raw) + 1023u) & ~1023u;
  const unsigned full0 = tc_smem(&bars[0]), empty0 = tc_smem(&bars[STAGES]), scored = tc_smem(&bars[2 * STAGES]);
  auto done = [&](int buf) { return tc_smem(&bars[2 * STAGES + 1 + buf]); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 16); mbar_init(empty0 + 8 * s, 1); }
    mbar_init(scored, 1);
    mbar_init(done(0), 1);
    mbar_init(done(1), 1);
    abort_s = 0;
    for (int h = 0; h < 8; ++h) marked_s[h] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int e = threadIdx.x; e < p.heads * NB; e += LC_THREADS) first_s[e / NB][e % NB] = LC_C;
  if (warp == LC_ISSUER) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    pdl_trigger();                                     // (not before: a kernel behind could take the tensor memory and wait for this one)
  }
  const int b = p.tile_seq[blockIdx.x], q0 = p.tile_q0[blockIdx.x], h0 = blockIdx.y * p.heads;
  const int qlen = p.cu_q_lens[b + 1] - p.cu_q_lens[b], t0 = p.cu_q_lens[b] + q0, n = min(LC_C, qlen - q0);
  const bool carry = p.context_lens[b] - qlen + q0 > 0;
  const int d = p.d, dv = p.dv, kd = (d + 31) / 32, kj = (n + 31) / 32;
  pdl_wait();
  LcTokens tokens;
  if (warp < p.heads) tokens = lc_tokens(p, t0, n, h0 + warp);       // (at most eight heads; used below)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_base_s;
  auto o_main = [&](int buf) { return tmem + 256 + buf * 2 * NB; };
  auto o_small = [&](int buf) { return NB <= 128 ? tmem + 256 + buf * 2 * NB + NB : tmem + 256; };
  const int N = (dv + 15) / 16 * 16;
  LcRing<STAGES> ring{full0, empty0};
  if (warp < LC_ISSUER) {
    // (a wait that runs out: the warp goes on through the loops and their barriers without work)
    const float* rq = p.rows + (size_t)t0 * p.row_stride + (size_t)(h0 / (p.H / p.G)) * d;
    const float* rk = rq + p.k_col;
    rq += p.q_col;
    const float* rv = p.values + (size_t)t0 * p.values_stride;
    auto one = [](int) { return 1.f; };
    {                                                  // the chunk's products q_i . k_j
      LcAlong<128> a, k;
      a.load(rq, p.row_stride, n, 0, d);
      k.load(rk, p.row_stride, n, 0, d);
      for (int s = 0; s < kd; ++s) {
        if (!ring.wait_empty(p, &abort_s)) break;
        const unsigned at = base + ring.slot() * STAGE;
        a.store(at, LC_A_BYTES, one);
        k.store(at + 2 * LC_A_BYTES, B_PART, one);
        if (s + 1 < kd) {
          a.load(rq, p.row_stride, n, 32 * (s + 1), d);
          k.load(rk, p.row_stride, n, 32 * (s + 1), d);
        }
        ring.give();
      }
    }
    if (warp < p.heads) {
      lc_sums(p, tokens, n, h0 + warp, Ls[warp], bs[warp]);
      __syncwarp();
#pragma unroll
      for (int e = 0; e < 4; ++e) fs[warp][4 * lane + e] = exp2f(Ls[warp].hi[4 * lane + e]);
    }
    asm volatile("bar.sync 1, 512;" ::: "memory");
    const int quarter = warp & 3, i = quarter * 32 + lane;      // the row this thread has in tensor memory
    const unsigned lane_off = (unsigned)(quarter * 32) << 16;
    auto epilogue = [&](int hh) {
      const int h = h0 + hh, buf = hh % BUFS;
      ring.ok = ring.ok && lc_wait_done(done(buf), (hh / BUFS) & 1, p, &abort_s);
      const int cols = ring.ok ? dv : 0;
      auto value = [&](int c0, float (&o)[32]) {
        unsigned m[32];
        tc_load32(o_main(buf) + lane_off + c0, m);
        if (NB <= 128) {
          unsigned s[32];
          tc_load32(o_small(buf) + lane_off + c0, s);
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __uint_as_float(m[e]) + __uint_as_float(s[e]);
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __uint_as_float(m[e]);
        }
        if (*(volatile int*)&marked_s[hh]) {           // rows from such a token on
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (i >= *(volatile int*)&first_s[hh][c0 + e]) o[e] = __int_as_float(0x7fffffff);
        }
      };
      if (!RETENTION) {
        const size_t row = ((size_t)(t0 + i) * p.H + h) * dv;
        for (int c0 = (warp >> 2) * 32; c0 < cols; c0 += 128) {
          float o[32];
          value(c0, o);
          if (i < n) {
#pragma unroll
            for (int e = 0; e < 32; e += 4)
              if (c0 + e < dv) *reinterpret_cast<float4*>(p.o_raw + row + c0 + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
          }
        }
      } else {
        // The rows go through the ring's memory (one head a CTA: every product that read it is done), so that a warp has a
        // row of the result: its sum of squares, its gate and its values side by side.
        float* tile = reinterpret_cast<float*>(lc_smem_raw + (base - tc_smem(lc_smem_raw)));      // (16-byte accesses)
        constexpr int TP = NB + 4;
        static_assert(LC_C * TP * sizeof(float) <= STAGES * STAGE, "the rows fit in the ring");
        for (int c0 = (warp >> 2) * 32; c0 < cols; c0 += LC_WORKERS / 4) {
          float o[32];
          value(c0, o);
#pragma unroll
          for (int e = 0; e < 32; e += 4) *reinterpret_cast<float4*>(tile + i * TP + c0 + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(LC_WORKERS) : "memory");
        for (int rr = warp; rr < n && cols > 0; rr += LC_ISSUER) {
          const TA* z = (const TA*)p.gate + (size_t)(t0 + rr) * p.gate_stride + (size_t)h * dv;
          TA* y = (TA*)p.out + ((size_t)(t0 + rr) * p.H + h) * dv;
          float4 o[(NB + 127) / 128], g[(NB + 127) / 128];
          float ss = 0.f;
#pragma unroll
          for (int u = 0; u < (NB + 127) / 128; ++u) {
            const int c = 128 * u + 4 * lane;
            if (c < dv) {
              g[u] = load4(z + c);
              o[u] = *reinterpret_cast<const float4*>(tile + rr * TP + c);
              ss += o[u].x * o[u].x + o[u].y * o[u].y + (o[u].z * o[u].z + o[u].w * o[u].w);
            }
          }
          const float f = rsqrtf(warp_sum(ss) / (float)dv + p.eps);
          auto act = [&](float x, float w) { return x * f * (w / (1.f + expf(-w))); };
#pragma unroll
          for (int u = 0; u < (NB + 127) / 128; ++u) {
            const int c = 128 * u + 4 * lane;
            if (c < dv) store4(y + c, make_float4(act(o[u].x, g[u].x), act(o[u].y, g[u].y), act(o[u].z, g[u].z), act(o[u].w, g[u].w)));
          }
        }
      }
    };
    for (int hh = 0; hh < p.heads; ++hh) {
      const int h = h0 + hh;
      if (BUFS == 1 && hh > 0) epilogue(hh - 1);       // its tensor memory is the next head's
      if (carry) {                                     // what the state before the chunk is worth to each row
        const float* S = p.scratch + ((size_t)blockIdx.x * p.H + h) * dv * d;
        LcAlong<128> a;
        LcAlong<NB> v;
        a.load(rq, p.row_stride, n, 0, d);
        v.load(S, d, dv, 0, d);
        for (int s = 0; s < kd; ++s) {
          if (!ring.wait_empty(p, &abort_s)) break;
          const unsigned at = base + ring.slot() * STAGE;
          a.store(at, LC_A_BYTES, [&](int r) { return fs[hh][r]; });
          v.store(at + 2 * LC_A_BYTES, B_PART, one);
          if (s + 1 < kd) {
            a.load(rq, p.row_stride, n, 32 * (s + 1), d);
            v.load(S, d, dv, 32 * (s + 1), d);
          }
          ring.give();
        }
      }
      if (hh == 0) ring.ok = ring.ok && lc_wait_done(scored, 0, p, &abort_s);
      LcAcross<NB> v;                                  // and the chunk's own tokens
      v.load(rv + (size_t)h * dv, p.values_stride, n, dv);
      const float Lhi = Ls[hh].hi[i], Llo = Ls[hh].lo[i];
      for (int s = 0; s < kj && ring.ok; ++s) {
        // this thread's eight scores of the step: row i, keys 32 s + 8 (warp / 4) ..
        unsigned m[8], x[8];
        const int j0 = 32 * s + (warp >> 2) * 8;
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(m[0]), "=r"(m[1]), "=r"(m[2]), "=r"(m[3]), "=r"(m[4]), "=r"(m[5]), "=r"(m[6]), "=r"(m[7]) : "r"(tmem + lane_off + j0));
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7]) : "r"(tmem + lane_off + 128 + j0));
        tc_wait_load();
        // (no branches: a masked key's power may overflow and is not taken; with them the eight powers came one after the other)
        float w[8], hi[8], lo[8], bj[8];
#pragma unroll
        for (int e = 0; e < 8; e += 4) {
          *reinterpret_cast<float4*>(hi + e) = *reinterpret_cast<const float4*>(Ls[hh].hi + j0 + e);
          *reinterpret_cast<float4*>(lo + e) = *reinterpret_cast<const float4*>(Ls[hh].lo + j0 + e);
          *reinterpret_cast<float4*>(bj + e) = *reinterpret_cast<const float4*>(bs[hh] + j0 + e);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float f = (__uint_as_float(m[e]) + __uint_as_float(x[e])) * (lc_power(Lhi, Llo, hi[e], lo[e]) * bj[e]);
          w[e] = j0 + e <= i ? f : 0.f;
        }
        if (!ring.wait_empty(p, &abort_s)) break;
        const unsigned at = base + ring.slot() * STAGE;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) lc_split(w[4 * c + e], hi[e], lo[e]);
          const unsigned to = at + i * 128 + (((2 * (warp >> 2) + c) ^ (i & 7)) << 4);
          lc_sts4(to, hi[0], hi[1], hi[2], hi[3]);
          lc_sts4(to + LC_A_BYTES, lo[0], lo[1], lo[2], lo[3]);
        }
        v.store(at + 2 * LC_A_BYTES, B_PART, one);
        if (v.take_out(at + 2 * LC_A_BYTES, B_PART, 32 * s + lane, first_s[hh])) { *(volatile int*)&marked_s[hh] = 1; __threadfence_block(); }
        if (s + 1 < kj) v.load(rv + (size_t)h * dv + (size_t)(32 * (s + 1)) * p.values_stride, p.values_stride, n - 32 * (s + 1), dv);
        ring.give();
      }
      if (BUFS == 2 && hh > 0) epilogue(hh - 1);
    }
    epilogue(p.heads - 1);
  } else if (lane == 0) {
    bool ok = true;
    for (int s = 0; s < kd && ok; ++s) {
      ok = ring.wait_full(p, &abort_s);
      if (!ok) break;
      const unsigned at = base + ring.slot() * STAGE;
      lc_step(tmem, tmem + 128, at, at + 2 * LC_A_BYTES, B_PART, lc_idesc(128), s == 0);
      ring.used();
    }
    tc_commit(scored);
    const unsigned idesc = lc_idesc(N);
    const int steps = (carry ? kd : 0) + kj;
    for (int hh = 0; hh < p.heads && ok; ++hh) {
      const int buf = hh % BUFS;
      for (int s = 0; s < steps; ++s) {
        ok = ring.wait_full(p, &abort_s);
        if (!ok) break;
        const unsigned at = base + ring.slot() * STAGE;
        lc_step(o_main(buf), o_small(buf), at, at + 2 * LC_A_BYTES, B_PART, idesc, s == 0);
        ring.used();
      }
      tc_commit(done(buf));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == LC_ISSUER) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---------------------------------------------------------------- launchers
// Floats of scratch: a state and a factor per chunk and head.
static long long lc_scratch(int tiles, int H, int d, int dv) { return (long long)tiles * H * ((long long)d * dv + 4); }

// Whether the kernels take these sizes and addresses.
static bool lc_supported(const LinearArgs& p) {
  auto on16 = [](const void* q) { return ((size_t)q % 16) == 0; };
  return p.d % 8 == 0 && p.d <= 256 && p.dv % 4 == 0 && p.dv <= 256 && p.row_stride % 4 == 0 && p.q_col % 4 == 0 && p.k_col % 4 == 0 &&
         p.values_stride % 4 == 0 && on16(p.values) && on16(p.rows) && on16(p.scratch) && on16(p.state) && (!p.o_raw || on16(p.o_raw)) && p.status;
}

template <typename K> static int lc_smem(K kernel, size_t bytes) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  return e == cudaSuccess ? GG_OK : gg_fail(GG_ERR_CUDA, "linear_chunks: %s", cudaGetErrorString(e));
}

template <int NB> static int lc_products(const LinearArgs& p, int num_tiles, cudaStream_t stream) {
  const size_t smem = 2 * (2 * LC_A_BYTES + 2 * NB * 128) + 1024;
  int rc = lc_smem(linear_products_kernel<NB>, smem);
  if (rc) return rc;
  gg_launch(linear_products_kernel<NB>, dim3(num_tiles, p.H / p.heads, (p.d + 127) / 128), dim3(LC_THREADS), smem, stream, p);
  return gg_check_launch("linear_products");
}
template <int NB, bool RETENTION, typename TA> static int lc_rows(const LinearArgs& p, int num_tiles, cudaStream_t stream) {
  const size_t smem = (NB > 128 ? 2 : 3) * (2 * LC_A_BYTES + 2 * (NB > 128 ? NB : 128) * 128) + 1024;
  int rc = lc_smem(linear_rows_kernel<NB, RETENTION, TA>, smem);
  if (rc) return rc;
  gg_launch(linear_rows_kernel<NB, RETENTION, TA>, dim3(num_tiles, p.H / p.heads), dim3(LC_THREADS), smem, stream, p);
  return gg_check_launch("linear_rows");
}

// The rows: a CTA takes one to eight heads of a group, so many that the machine is done soonest.  A chunk's products q_i . k_j take a
// CTA about as long as 0.8 of a head (10 k clocks of 12 k), and one CTA fits on a multiprocessor: 64 heads of a group and 16 chunks as
// 128 CTAs of eight heads 92 us, as 256 of four 101; 16 heads on 4 groups as 128 CTAs of two 37, as 256 of one 45.  With values of 16 to
// 256, keys of 32 to 256, 8 to 128 heads on 1 to 32 groups and 256 to 4096 tokens no step of 84 became slower by this choice than with as
// many heads as left 222 CTAs (0.74 to 1.00 of its time, the shorter arithmetic of the decays included).
template <bool RETENTION, typename TA> static int lc_all_rows(LinearArgs p, int num_tiles, cudaStream_t stream) {
  p.heads = 1;
  auto turns = [&](int heads) { return ((long long)num_tiles * (p.H / heads) + 147) / 148 * (4 + 5 * heads); };
  for (int heads = 2; heads <= 8 && p.H / p.G % heads == 0; heads *= 2)
    if (turns(heads) < turns(p.heads)) p.heads = heads;
  if (p.dv <= 64) return lc_rows<64, RETENTION, TA>(p, num_tiles, stream);
  if (p.dv <= 128) return lc_rows<128, RETENTION, TA>(p, num_tiles, stream);
  return lc_rows<256, RETENTION, TA>(p, num_tiles, stream);
}

template <bool RETENTION, typename TA> static int lc_run(LinearArgs p, int num_tiles, cudaStream_t stream) {
  p.tiles = num_tiles;
  p.factor = p.scratch + (long long)num_tiles * p.H * p.d * p.dv;
  const int rep = p.H / p.G;
  // the chunks' products: heads of a group side by side, up to 256 columns (eight neighbouring ones are of one head)
  p.heads = 1;
  while (p.heads < 8 && p.dv % 8 == 0 && rep % (2 * p.heads) == 0 && 2 * p.heads * p.dv <= 256) p.heads *= 2;
  const int cols = p.heads * p.dv;
  int rc = cols <= 64 ? lc_products<64>(p, num_tiles, stream) : cols <= 128 ? lc_products<128>(p, num_tiles, stream) : lc_products<256>(p, num_tiles, stream);
  if (rc) return rc;
  gg_launch(linear_scan_kernel, dim3(p.B, p.H, (p.d * p.dv / 4 + 255) / 256), dim3(256), 0, stream, p);
  rc = gg_check_launch("linear_scan");
  if (rc) return rc;
  return lc_all_rows<RETENTION, TA>(p, num_tiles, stream);
}

// gg_delta_recur's plain recurrence over the sequences whose chunks of 128 tokens are the tiles (all chunks of a sequence, in
// their order); the others are left alone.  Returns GG_ERR_UNSUPPORTED, and launches nothing, where sizes or addresses are not
// for these kernels.  Scratch the caller provides: float[num_tiles * H * (d * dv + 4)].
extern "C" int gg_linear_chunks(const float* qkv, const float* beta, const float* decay, float* state, float* scratch,
                                long long scratch_floats, const int* tile_seq, const int* tile_q0, int num_tiles,
                                const int* cu_q_lens, const int* context_lens, const int* state_slots, int T, int B, int G, int H,
                                int d, int dv, float* o_raw, int* status, cudaStream_t stream) {
  GG_REQUIRE(T >= 0 && B > 0 && G > 0 && H > 0 && H % G == 0 && d > 0 && dv > 0 && num_tiles >= 0, "linear_chunks: bad sizes T=%d B=%d G=%d H=%d d=%d dv=%d", T, B, G, H, d, dv);
  GG_REQUIRE(qkv && beta && decay && state && scratch && o_raw && status, "linear_chunks: a pointer is null");
  LinearArgs p = {};
  p.rows = qkv; p.row_stride = 2ll * G * d + (long long)H * dv; p.q_col = 0; p.k_col = G * d; p.values = qkv + 2 * G * d; p.values_stride = p.row_stride;
  p.beta = beta; p.decay = decay; p.state = state; p.scratch = scratch; p.tile_seq = tile_seq; p.tile_q0 = tile_q0;
  p.cu_q_lens = cu_q_lens; p.context_lens = context_lens; p.state_slots = state_slots;
  p.B = B; p.G = G; p.H = H; p.d = d; p.dv = dv; p.o_raw = o_raw; p.status = status;
  if (!lc_supported(p) || H > 65535) return GG_ERR_UNSUPPORTED;
  GG_REQUIRE(scratch_floats >= lc_scratch(num_tiles, H, d, dv), "linear_chunks: scratch of %lld values is too small", scratch_floats);
  if (num_tiles == 0) return GG_OK;
  return lc_run<false, float>(p, num_tiles, stream);
}

// Retention's prompt portions (see retention.cu): rows of gg_retention_rows, one fixed decay a head, unit norm and gate.
extern "C" int gg_linear_retention(const float* rows, const float* log2_decay, float* state, float* scratch, long long scratch_floats,
                            const int* tile_seq, const int* tile_q0, int num_tiles, const int* cu_q_lens, const int* context_lens,
                            const int* state_slots, int T, int B, const void* gate, long long gate_stride, float eps, int H, int d,
                            int dv, int dtype, void* out, int* status, cudaStream_t stream) {
  GG_REQUIRE(T >= 0 && B > 0 && H > 0 && d > 0 && dv > 0 && num_tiles >= 0, "linear_retention: bad sizes T=%d B=%d H=%d d=%d dv=%d", T, B, H, d, dv);
  GG_REQUIRE(rows && log2_decay && state && scratch && gate && out && status && gate_stride >= (long long)H * dv, "linear_retention: bad arguments");
  LinearArgs p = {};
  p.rows = rows; p.row_stride = (long long)H * (2 * d + dv); p.q_col = 0; p.k_col = H * d; p.values = rows + 2 * H * d; p.values_stride = p.row_stride;
  p.log2_decay = log2_decay; p.state = state; p.scratch = scratch; p.tile_seq = tile_seq; p.tile_q0 = tile_q0;
  p.cu_q_lens = cu_q_lens; p.context_lens = context_lens; p.state_slots = state_slots;
  p.B = B; p.G = H; p.H = H; p.d = d; p.dv = dv;
  p.gate = gate; p.gate_stride = gate_stride; p.eps = eps; p.out = out; p.status = status;
  if (!lc_supported(p) || (dtype != GG_F32 && dtype != GG_BF16) || gate_stride % 4 || ((size_t)gate % 16) || ((size_t)out % 16) || H > 65535)
    return GG_ERR_UNSUPPORTED;
  GG_REQUIRE(scratch_floats >= lc_scratch(num_tiles, H, d, dv), "linear_retention: scratch of %lld values is too small", scratch_floats);
  if (num_tiles == 0) return GG_OK;
  return dtype == GG_F32 ? lc_run<true, float>(p, num_tiles, stream) : lc_run<true, __nv_bfloat16>(p, num_tiles, stream);
}
