// Token selection from float32 logits, one thread block per row.
//
// Follows internal/engine/sampling.go:40-192 of the reference (which samples on
// the host in float64): temperature <= 1e-9 means greedy (first maximum wins);
// otherwise logits/T, keep the top_k largest (0 = off), softmax, keep the
// smallest sorted prefix whose mass reaches top_p (0 or >= 1 = off), renormalise,
// and take the first index whose running sum exceeds a uniform draw.  The draw
// of request r for its n-th token is a counter-based hash of (seed_r, n), so a
// request's tokens do not depend on what else is in the batch.
// Elements equal to the top-k or top-p threshold value are all kept.
#include "common.cuh"
#include <cstring>
#include <cstdlib>

#define SAMPLE_THREADS 1024

__device__ __forceinline__ unsigned int ordered_key(float x) {
  const unsigned int b = __float_as_uint(x);
  return b ^ ((unsigned int)((int)b >> 31) | 0x80000000u);
}

__device__ __forceinline__ float uniform_draw(unsigned long long seed, unsigned long long n) {
  unsigned long long z = seed + (n + 1ULL) * 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  z = z ^ (z >> 31);
  return (float)(z >> 40) * (1.0f / 16777216.0f);
}

// Which values of a row a thread has: four neighbouring ones from 4 start on, every 4 stride further.  Two blocks that share a row
// have the threads of one twice as large between them.  AHEAD: how many pairs of loads are on their way beside the pair at hand;
// 0: eight loads at a time, for a pass of a few instructions a value alone (argmax of 128 k: 5.0 us, with pairs of loads 7.5).
template <int AHEAD = 1> struct Walk { int start, stride; };

// f(i, v, there) for every four values v at row[4 i] that are this thread's, by whole warps (there: inside the row).  A pass runs its
// loop a few times only and the code of an unrolled one comes from L2 too: two loads a turn and the next ones on their way take 20
// thousand clocks of 128 k values with exponentials, sixteen loads a turn 42.
template <int AHEAD, typename F> __device__ __forceinline__ void each_four(const float* row, int V4, const Walk<AHEAD> walk, F&& f) {
  const float4* row4 = reinterpret_cast<const float4*>(row);
  const int lane = threadIdx.x & 31, step = 2 * walk.stride;
  if constexpr (AHEAD == 0) {
    for (int i = walk.start; i < V4; i += 8 * walk.stride) {       // (f takes no part in warps)
      float4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i + u * walk.stride < V4) v[u] = row4[i + u * walk.stride];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i + u * walk.stride < V4) f(i + u * walk.stride, v[u], true);
    }
    return;
  }
  float4 v[AHEAD + 1][2];
#pragma unroll
  for (int a = 0; a <= AHEAD; ++a)
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (walk.start + a * step + u * walk.stride < V4) v[a][u] = row4[walk.start + a * step + u * walk.stride];
#pragma unroll 1
  for (int i = walk.start; i - lane < V4; i += step) {
    const float4 c[2] = {v[0][0], v[0][1]};
#pragma unroll
    for (int a = 0; a < AHEAD; ++a) { v[a][0] = v[a + 1][0]; v[a][1] = v[a + 1][1]; }
    const int n = i + (AHEAD + 1) * step;
    if (n < V4) v[AHEAD][0] = row4[n];
    if (n + walk.stride < V4) v[AHEAD][1] = row4[n + walk.stride];
#pragma unroll
    for (int u = 0; u < 2; ++u) f(i + u * walk.stride, c[u], i + u * walk.stride < V4);
  }
}

// Of the threads' maxima and their first indices the block's.
__device__ __forceinline__ int first_of_block(float best, int bi, float* red_f, int* red_i, float* max_out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  __syncthreads();
  if (lane == 0) { red_f[warp] = best; red_i[warp] = bi; }
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    best = lane < nw ? red_f[lane] : -INFINITY;
    bi = lane < nw ? red_i[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) { red_f[32] = best; red_i[32] = bi; }
  }
  __syncthreads();
  if (max_out) *max_out = red_f[32];
  return red_i[32];
}

// First index of the maximum of row[0..V) (0x7fffffff: none above -infinity).  own: the maximum of this thread's values.
template <int AHEAD = 1>
__device__ int block_argmax(const float* row, int V, float* red_f, int* red_i, float* max_out, float* own = nullptr,
                            const Walk<AHEAD> walk = {(int)threadIdx.x, (int)blockDim.x}) {
  float best = -INFINITY;
  int bi = 0x7fffffff;
  if ((((size_t)row) & 15) == 0) {
    // within a thread indices only grow, so ">" keeps the first maximum
    const int V4 = V >> 2;
    each_four(row, V4, walk, [&](int i, const float4& v, bool there) {
      if (there) {
        if (v.x > best) { best = v.x; bi = 4 * i; }
        if (v.y > best) { best = v.y; bi = 4 * i + 1; }
        if (v.z > best) { best = v.z; bi = 4 * i + 2; }
        if (v.w > best) { best = v.w; bi = 4 * i + 3; }
      }
    });
    for (int i = (V4 << 2) + walk.start; i < V; i += walk.stride) {
      const float v = row[i];
      if (v > best || (v == best && i < bi)) { best = v; bi = i; }
    }
  } else {
    for (int i = walk.start; i < V; i += walk.stride) {
      const float v = row[i];
      if (v > best || (v == best && i < bi)) { best = v; bi = i; }
    }
  }
  if (own) *own = best;
  return first_of_block(best, bi, red_f, red_i, max_out);
}
__device__ __forceinline__ int first_if_none(int i) { return i == 0x7fffffff ? 0 : i; }

__global__ void argmax_kernel(const float* __restrict__ logits, int V, int* __restrict__ out) {
  __shared__ float red_f[33];
  __shared__ int red_i[33];
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x;
  const int idx = first_if_none(block_argmax<0>(logits + (size_t)r * V, V, red_f, red_i, nullptr, nullptr, Walk<0>{(int)threadIdx.x, SAMPLE_THREADS}));
  if (threadIdx.x == 0) out[r] = idx;
}

// Radix descent from the most significant byte: the key K such that the elements
// with key > K weigh less than `target` and those with key >= K weigh at least
// `target`.  weight(i) = 1 (count mode, the k-th largest) or exp((x_i - m) * invT)
// (mass mode).  Only elements with key >= floor_key take part.
// Leading byte: logits crowd into a few of its values (one shared histogram with atomics
// serialised there: a millisecond per row at a vocabulary of 128 k), and the threshold is
// almost always within the three values at and below the maximum's.  So a thread first adds up,
// in registers, the weights of its elements from the lower border of each of those three bins
// on, and the block adds the threads' sums in a fixed order.  Only if all three together do not
// reach the target is the leading byte binned in full.  Lower bytes (and that full pass): the
// elements still in the range spread over many bins; weights in fixed point (40 fraction bits),
// added atomically as three 32-bit pieces a bin, or as 64-bit integers where a row has so many
// values that a piece could overflow (FX_MAX_VALUES).  Integer sums do not depend on their order
// and the others have a fixed one, so the result is the same on every run.
// ---- a row spread over the CTAs of a thread-block cluster (sample_cluster_kernel): what a
// CTA shows its neighbours.  Two copies, used in turn: a copy is written again only after a
// further cluster barrier, which nobody passes before everybody has read the one before.
struct ClusterPub {
  float hist[2][256];
  float f[2];
  int i[2];
  int parity;            // which copy the next exchange uses (the same in every CTA)
};
__device__ __forceinline__ unsigned sc_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned sc_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void sc_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <typename T> __device__ __forceinline__ T sc_load(const T* local, unsigned rank) {
  unsigned v, a = (unsigned)__cvta_generic_to_shared(local);
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %1, %2;\n\t"
      "ld.shared::cluster.b32 %0, [ra];\n\t}"
      : "=r"(v) : "r"(a), "r"(rank) : "memory");
  T out;
  memcpy(&out, &v, 4);
  return out;
}

// f(x) for the values of row[0..V) that are this thread's.
template <int AHEAD, typename F> __device__ __forceinline__ void each_value(const float* row, int V, const Walk<AHEAD> walk, F&& f) {
  const int V4 = (((size_t)row) & 15) == 0 ? V >> 2 : 0;
  each_four(row, V4, walk, [&](int, const float4& v, bool there) {
    if (there) { f(v.x); f(v.y); f(v.z); f(v.w); }
  });
  for (int i = (V4 << 2) + walk.start; i < V; i += walk.stride) f(row[i]);
}

// The values of row[0..V) with keys in [lo, hi] that are this block's to keep[0..room), in no particular order; *n = how many there
// are (also those beyond the room).  A warp adds the hits of four values a lane to *n at once, then writes them value by value: the
// lanes that hit write side by side (each lane writing its own hits in a row met a bank eight times over: 41 us of a row with 27 k
// hits among 128 k).
template <int AHEAD>
__device__ void collect(const float* row, int V, const Walk<AHEAD> walk, float* keep, int room, int* n, unsigned lo, unsigned hi) {
  if (threadIdx.x == 0) *n = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int V4 = (((size_t)row) & 15) == 0 ? V >> 2 : 0;
  auto in = [&](float x) { const unsigned k = ordered_key(x); return k >= lo && k <= hi; };
  const int first = walk.start - lane;                   // (the warp's; lanes are neighbours)
  each_four(row, V4, walk, [&](int, const float4& v, bool there) {
    const float f[4] = {v.x, v.y, v.z, v.w};
    unsigned m[4], all = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) { m[j] = __ballot_sync(0xffffffffu, there && in(f[j])); all |= m[j]; }
    if (!all) return;
    int at = 0;
    if (lane == 0) at = atomicAdd(n, __popc(m[0]) + __popc(m[1]) + (__popc(m[2]) + __popc(m[3])));
    at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int to = at + __popc(m[j] & below);
      if ((m[j] >> lane & 1u) && to < room) keep[to] = f[j];
      at += __popc(m[j]);
    }
  });
  for (int b = (V4 << 2) + first; b < V; b += walk.stride) {
    const int i = b + lane;
    const bool hit = i < V && in(row[i]);
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    int at = 0;
    if (lane == 0 && m) at = atomicAdd(n, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & below);
    if (hit && at < room) keep[at] = row[i];
  }
  __syncthreads();
}

// ---- a row shared by the two blocks of a cluster (sample_kernel<2>): each has half of the threads that one block alone has, does what
// those do, and tells the other what they found, so that every sum is formed from the same numbers in the same order.  What is told
// goes to the other's copy, one of two in turn: a copy is written again only after a further cluster barrier.
struct PairPub {
  float f[2][4][32];
  int i[2][2];
  unsigned long long bins[2][256];
};
__device__ __forceinline__ unsigned pair_addr(const void* local) {        // of the same variable in the other block
  unsigned v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(v) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(sc_rank() ^ 1u));
  return v;
}
__device__ __forceinline__ void pair_tell(float* to, float v) {
  *to = v;
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(pair_addr(to)), "f"(v) : "memory");
}
__device__ __forceinline__ void pair_tell(int* mine, int* others, int v) {
  *mine = v;
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(pair_addr(others)), "r"(v) : "memory");
}
// block_sum of N values over both blocks' 32 warps
template <int N> __device__ __forceinline__ void pair_sums(float (&v)[N], PairPub* pub, int& par) {
  const int lane = threadIdx.x & 31, slot = sc_rank() * (blockDim.x >> 5) + (threadIdx.x >> 5);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    v[j] = warp_sum(v[j]);
    if (lane == 0) pair_tell(&pub->f[par][j][slot], v[j]);
  }
  sc_barrier();
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = warp_sum(pub->f[par][j][lane]);
  par ^= 1;
}
// the sum of both blocks' v (of thread 0); *mine: this block's
__device__ __forceinline__ int pair_count(int v, PairPub* pub, int& par) {
  if (threadIdx.x == 0) pair_tell(&pub->i[par][0], &pub->i[par][1], v);
  sc_barrier();
  const int s = pub->i[par][0] + pub->i[par][1];
  par ^= 1;
  return s;
}

// Sums of weights in fixed point (40 fraction bits) in bins of shared memory.  A 64-bit atomic on shared memory is a loop
// of compare-and-swap, so a weight is added in three pieces of 14 bits, 32-bit atomics that the memory does itself; the
// pieces of up to 2^18 weights cannot overflow (longer rows add 64 bits at a time), and the total is the same integer.
#define FX_ONE 1099511627776.f           // 2^40
#define FX_PIECES 3
__device__ __forceinline__ unsigned long long fixed_weight(float w) { return (unsigned long long)(w * FX_ONE); }
__device__ __forceinline__ void add_bin(unsigned* bin, unsigned v) {      // (bin is in shared memory: no generic address to resolve)
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bin)), "r"(v) : "memory");
}
__device__ __forceinline__ void add_fixed(unsigned* bins, int stride, int bin, unsigned long long w) {
#pragma unroll
  for (int k = 0; k < FX_PIECES; ++k) {
    const unsigned piece = (unsigned)(w >> (14 * k)) & (k + 1 < FX_PIECES ? 0x3fffu : 0xffffffffu);
    if (piece) add_bin(bins + k * stride + bin, piece);
  }
}
__device__ __forceinline__ unsigned long long fixed_sum(const unsigned* bins, int stride, int bin) {
  unsigned long long s = 0;
#pragma unroll
  for (int k = 0; k < FX_PIECES; ++k) s += (unsigned long long)bins[k * stride + bin] << (14 * k);
  return s;
}
#define FX_MAX_VALUES (1 << 18)

// The first bin from the top of hist[0..256) whose weight, added to `above` and to that of the bins over it, reaches
// target (bin 0 where none does), and the weight over it, to hist[256] and hist[257].  Called by one warp.  Lane l takes
// bins 255 - 8 l down to 248 - 8 l: one thread walking 256 bins is 256 dependent reads of shared memory, 4 us a pass.
__device__ __forceinline__ void pick_bin(float* hist, float above, float target) {
  const int lane = threadIdx.x & 31;
  float hs[8], s = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int b = 255 - 8 * lane - j;
    hs[j] = b > 0 ? hist[b] : 0.f;
    s += hs[j];
  }
  float incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  float cum = above + (incl - s);
  int fb = -1;
  float fcum = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int b = 255 - 8 * lane - j;
    if (b > 0 && fb < 0) {
      if (cum + hs[j] >= target) { fb = b; fcum = cum; }
      else cum += hs[j];
    }
  }
  const unsigned any = __ballot_sync(0xffffffffu, fb >= 0);
  const int src = any ? __ffs(any) - 1 : 31;
  const int bin = any ? __shfl_sync(0xffffffffu, fb, src) : 0;
  const float all = __shfl_sync(0xffffffffu, incl, 31);
  const float cumv = any ? __shfl_sync(0xffffffffu, fcum, src) : above + all;
  if (lane == 0) {
    hist[256] = cumv;
    hist[257] = __int_as_float(bin);
  }
}

// MODE 1: row is this CTA's part of the row and the histogram of a pass is the sum over the
// cluster's CTAs in rank order, the same in every CTA, so every CTA descends alike.  MODE 2: the two blocks of a pair walk the row
// (or their own lists of what is left of it) together.  last: the lowest bit of the byte it ends with.
// bins: FX_PIECES * 256 integers, 8-byte aligned.  unordered: row is a copy whose order differs from run to run, so the
// float32 sums of the first pass are left out.  sum_of_all: target is share times the sum of all weights, which the first
// pass makes too.  keep, keep_n: where given (room for keep_room values; not MODE 1), what is left of the row once
// the leading byte is known is copied there, and the lower bytes' passes read the copy.
template <bool MASS, int MODE, int AHEAD = 1>
__device__ unsigned int radix_threshold(const float* row, int V, float m, float invT,
                                        unsigned int floor_key, float target, float* hist,
                                        float* red, unsigned* bins, ClusterPub* pub = nullptr,
                                        float* keep = nullptr, int* keep_n = nullptr, int keep_room = 0, const bool sum_of_all = false,
                                        float share = 0.f, const bool unordered = false,
                                        Walk<AHEAD> walk = {(int)threadIdx.x, (int)blockDim.x}, PairPub* pair = nullptr, int* turn = nullptr, const int last = 0) {
  constexpr bool CL = MODE == 1;
  const int warp = threadIdx.x >> 5;
  unsigned int prefix = 0, pmask = 0;
  float above = 0.f;       // weight of keys strictly above the current prefix range
  // hist[0..n) = the block's (CL: the cluster's) sum of hist[0..n) as every thread sees it
  auto exchange = [&](int n) {
    if (CL) {
      const int par = pub->parity;
      for (int i = threadIdx.x; i < n; i += blockDim.x) pub->hist[par][i] = hist[i];
      sc_barrier();                            // (also a barrier of the CTA)
      const unsigned C = sc_size();
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        float v = 0.f;
        for (unsigned c = 0; c < C; ++c) v += sc_load(&pub->hist[par][i], c);
        hist[i] = v;
      }
      __syncthreads();
      if (threadIdx.x == 0) pub->parity = par ^ 1;
    }
    __syncthreads();
  };
  // ---- leading byte, the three bins at and below the maximum's
  const int top = (int)(ordered_key(m) >> 24);
  bool full = true;                            // the leading byte still has to be binned in full
  if (!unordered) {
    // the weight of the values from the lower border of each of the three bins on
    const unsigned b0 = (unsigned)top << 24, b1 = (unsigned)max(top - 1, 0) << 24, b2 = (unsigned)max(top - 2, 0) << 24;
    float acc0 = 0.f, acc1 = 0.f, acc2 = 0.f, all = 0.f;
    each_value(row, V, walk, [&](float x) {
      // (without branches: a value's chain of steps then runs beside its neighbours'; adding 0 changes no sum)
      const unsigned int k = ordered_key(x);
      if (MASS) {
        const float e = expf((x - m) * invT);
        const float w = k < floor_key ? 0.f : e;
        acc0 += k >= b0 ? w : 0.f;
        acc1 += k >= b1 ? w : 0.f;
        acc2 += k >= b2 ? w : 0.f;
        all += w;
      } else if (k >= floor_key && k >= b2) {           // (few do)
        if (k >= b0) acc0 += 1.f;
        if (k >= b1) acc1 += 1.f;
        acc2 += 1.f;
      }
    });
    if constexpr (MODE == 2) {
      float v[4] = {acc0, acc1, acc2, all};
      pair_sums(v, pair, *turn);
      acc0 = v[0]; acc1 = v[1]; acc2 = v[2];
      if (sum_of_all) target = share * v[3];
    } else {
      if (sum_of_all) target = share * block_sum(all, red);     // the target is a share of the sum
      acc0 = block_sum(acc0, red);
      acc1 = block_sum(acc1, red);
      acc2 = block_sum(acc2, red);
    }
    if (threadIdx.x == 0) { hist[0] = acc0; hist[1] = acc1; hist[2] = acc2; }
    __syncthreads();
    exchange(3);
    for (int d = 0; d <= 2 && d <= top; ++d) {
      if (hist[d] >= target) {
        prefix = (unsigned int)(top - d) << 24;
        pmask = 255u << 24;
        above = d > 0 ? hist[d - 1] : 0.f;
        full = false;
        break;
      }
    }
    __syncthreads();                           // hist is written again below
  }
  for (int shift = full ? 24 : 16; shift >= last; shift -= 8) {
    const bool wide = MASS && V > FX_MAX_VALUES;
    unsigned long long* bins64 = reinterpret_cast<unsigned long long*>(bins);
    if (!CL && keep && pmask == 255u << 24 && shift == 16) {
      // the values that share the threshold's leading byte (their order is as they come: the sums are integers)
      collect(row, V, walk, keep, keep_room, keep_n, max(floor_key, prefix), prefix | 0xffffffu);
      int left = *keep_n;
      if constexpr (MODE == 2) left = pair_count(left, pair, *turn);
      if (left <= keep_room) {
        row = keep;
        V = *keep_n;
        if constexpr (MODE == 2) walk = {(int)threadIdx.x, (int)blockDim.x};
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < FX_PIECES * 256; i += blockDim.x) bins[i] = 0u;
    __syncthreads();
    each_value(row, V, walk, [&](float x) {
      const unsigned int k = ordered_key(x);
      if (k >= floor_key && (k & pmask) == prefix) {
        if (wide) atomicAdd(bins64 + ((k >> shift) & 255u), fixed_weight(expf((x - m) * invT)));
        else if (MASS) add_fixed(bins, 256, (k >> shift) & 255u, fixed_weight(expf((x - m) * invT)));
        else add_bin(bins + ((k >> shift) & 255u), 1u);
      }
    });
    __syncthreads();
    if constexpr (MODE == 2) {
      const int par = *turn;
      unsigned long long own = 0;
      const int i = threadIdx.x;                       // (512 threads)
      if (i < 256) {
        own = !MASS ? bins[i] : wide ? bins64[i] : fixed_sum(bins, 256, i);
        asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(pair_addr(&pair->bins[par][i])), "l"(own) : "memory");
      }
      sc_barrier();
      if (i < 256) {
        own += pair->bins[par][i];
        hist[i] = MASS ? (float)own * (1.f / FX_ONE) : (float)own;
      }
      __syncthreads();
      *turn = par ^ 1;
    } else {
      for (int i = threadIdx.x; i < 256; i += blockDim.x)
        hist[i] = MASS ? (float)(wide ? bins64[i] : fixed_sum(bins, 256, i)) * (1.f / FX_ONE) : (float)bins[i];
      __syncthreads();
      exchange(256);
    }
    if (warp == 0) pick_bin(hist, above, target);
    __syncthreads();
    above = hist[256];
    const unsigned int bin = (unsigned int)__float_as_int(hist[257]);
    prefix |= bin << shift;
    pmask |= 255u << shift;
    __syncthreads();
  }
  return prefix;
}

// A CTA a row.  Bound by what one multiprocessor reads of a row from L2 (4 us for 128 k values) and by the chain of block-
// wide steps, so the row is walked as few times as possible: the maximum; the values that can be among the top_k largest
// (those above the k-th largest of the threads' own maxima, some hundreds), or one pass for the sum and the leading byte
// of top_p and one that copies the values of that byte to shared memory (`room` of them; what does not fit is walked where
// it is); the sums in index order.  What bounds it: the chain of passes, each a few turns of a loop by 16 or 32 warps, whose code
// arrives from L2 too (each_four).  128 k values, 148 rows: 41 us with top_k, 90 with top_p alone (before loops of two loads: 55, 117).
// BLOCKS = 2: the row on two multiprocessors, each with half of the threads (PairPub); the same numbers in the same order.  64 rows, us
// without thresholds, with top_k, with top_p alone, with both; two multiprocessors a row / one: 128 k values 21 / 26, 33 / 37, 58 / 85,
// 44 / 52; 32 k 10.4 / 11.3, 21 / 22, 26 / 33, 31 / 33; 16384 (the fewest) 8.6 / 8.6, 18.7 / 19.2, 19.8 / 23.4, 26.9 / 28.4; 38 and 74
// rows alike.
template <int BLOCKS>
__global__ void __launch_bounds__(SAMPLE_THREADS / BLOCKS)
sample_kernel(const float* __restrict__ logits, int V, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const unsigned long long* __restrict__ seeds,
              const unsigned long long* __restrict__ draw_index, int* __restrict__ out, int room) {
  constexpr int THREADS = SAMPLE_THREADS / BLOCKS, AHEAD = BLOCKS == 2 ? 3 : 1, MODE = BLOCKS == 2 ? 2 : 0;
  extern __shared__ __align__(16) float keep[];          // [room]
  __shared__ float red_f[33];
  __shared__ int red_i[33];
  __shared__ float hist[258];
  __shared__ __align__(8) unsigned bins[FX_PIECES * 256];
  __shared__ float scan[SAMPLE_THREADS / 32 + 1];
  __shared__ int keep_n;
  __shared__ int found, other_found;
  __shared__ unsigned long long sum64;
  __shared__ PairPub pub_s;
  PairPub* pub = &pub_s;
  int turn = 0;
  const int rank = BLOCKS == 2 ? (int)sc_rank() : 0, tid = rank * THREADS + threadIdx.x;       // the thread's place in the row
  const Walk<AHEAD> walk = {tid, SAMPLE_THREADS};
  const Walk<AHEAD> local = {(int)threadIdx.x, THREADS};
  pdl_trigger();
  if constexpr (BLOCKS == 2) sc_barrier();               // the other block's memory is there
  pdl_wait();
  const int r = BLOCKS == 2 ? blockIdx.y : blockIdx.x;
  const float* row = logits + (size_t)r * V;
  const float T = temperature[r];
  float m, own;
  int amax;
  if constexpr (BLOCKS == 2) amax = block_argmax(row, V, red_f, red_i, &m, &own, walk);
  else amax = block_argmax<0>(row, V, red_f, red_i, &m, &own, Walk<0>{tid, SAMPLE_THREADS});
  if constexpr (BLOCKS == 2) {
    float* f = &pub->f[0][0][0];
    if (threadIdx.x == 0) {
      pair_tell(f + rank, m);
      asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(pair_addr(&pub->i[0][1])), "r"(amax) : "memory");
    }
    sc_barrier();
    const float om = f[rank ^ 1];
    const int oi = pub->i[0][1];
    if (om > m || (om == m && oi < amax)) amax = oi;
    m = fmaxf(m, om);                                    // (a NaN is never a maximum here)
    turn = 1;
  }
  amax = first_if_none(amax);
  if (T <= 1e-9f) {
    if (tid == 0) out[r] = amax;
    return;
  }
  const float invT = 1.f / T;
  const int lane = threadIdx.x & 31, warp = tid >> 5;
  unsigned int floor_key = 0;
  const int k = top_k ? top_k[r] : 0;
  const float p = top_p ? top_p[r] : 0.f;
  bool kept = false;                                     // keep[0 .. keep_n) holds every value that can still be drawn
  int kept_n = 0;
  if (k > 0 && k < V) {
    if (k <= SAMPLE_THREADS && room >= SAMPLE_THREADS) {
      keep[tid] = own;
      if constexpr (BLOCKS == 2) {
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(pair_addr(keep + tid)), "f"(own) : "memory");
        sc_barrier();
        turn ^= 1;
      } else {
        __syncthreads();
      }
      // (sixteen bits of it: what they leave in below the k-th largest is gone with the threshold itself)
      const unsigned pivot = radix_threshold<false, 0, AHEAD>(keep, SAMPLE_THREADS, m, invT, 0u, (float)k, hist, red_f, bins, nullptr, nullptr,
                                                              nullptr, 0, false, 0.f, false, local, nullptr, nullptr, 16);
      __syncthreads();
      if constexpr (BLOCKS == 2) sc_barrier();           // (both have read what each told the other)
      collect(row, V, walk, keep, room, &keep_n, pivot, 0xffffffffu);    // at least k values: k threads have one
      kept_n = keep_n;
      if constexpr (BLOCKS == 2) kept_n = pair_count(kept_n, pub, turn);
      kept = kept_n <= room;
      if (BLOCKS == 2 && kept) {                         // the other's behind this block's: both have them all
        const int mine = keep_n;
        for (int i = threadIdx.x; i < kept_n - mine; i += THREADS) keep[mine + i] = sc_load(keep + i, rank ^ 1);
        __syncthreads();
      }
    }
    floor_key = kept ? radix_threshold<false, 0, AHEAD>(keep, kept_n, m, invT, 0u, (float)k, hist, red_f, bins, nullptr, nullptr, nullptr, 0,
                                                    false, 0.f, false, local)
                     : radix_threshold<false, MODE, AHEAD>(row, V, m, invT, 0u, (float)k, hist, red_f, bins, nullptr, keep, &keep_n, room,
                                                       false, 0.f, false, walk, pub, &turn);
  }
  if (p > 0.f && p < 1.f) {
    if (kept) {
      // the copy's order differs from run to run: integer sums only
      if (threadIdx.x == 0) sum64 = 0ULL;
      __syncthreads();
      unsigned long long z = 0;
      for (int i = threadIdx.x; i < kept_n; i += THREADS)
        if (ordered_key(keep[i]) >= floor_key) z += fixed_weight(expf((keep[i] - m) * invT));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
      if (lane == 0 && z) atomicAdd(&sum64, z);
      __syncthreads();
      floor_key = radix_threshold<true, 0, AHEAD>(keep, kept_n, m, invT, floor_key, p * ((float)sum64 * (1.f / FX_ONE)), hist, red_f, bins,
                                              nullptr, nullptr, nullptr, 0, false, 0.f, true, local);
    } else {
      floor_key = radix_threshold<true, MODE, AHEAD>(row, V, m, invT, floor_key, 0.f, hist, red_f, bins, nullptr, keep, &keep_n, room, true, p,
                                                 false, walk, pub, &turn);
    }
  }
  // Running sum in index order over the values that are left: a warp owns a stretch of the row and sums it in up to 32
  // blocks, whose sums its lanes keep; the block that holds the draw is then walked 128 values at a time.
  const int seg = ((V + SAMPLE_THREADS * 4 - 1) / (SAMPLE_THREADS * 4)) * 128;
  const int blk = max(512, ((seg + 31) / 32 + 127) / 128 * 128);
  const int s0 = min(V, warp * seg), s1 = min(V, s0 + seg);
  const bool vec = (((size_t)row) & 15) == 0;
  auto values4 = [&](int i, float (&x)[4]) {             // values i .. i + 3 (past the stretch: none)
    if (vec && i + 4 <= s1) {
      const float4 v = *reinterpret_cast<const float4*>(row + i);
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = i + j < s1 ? row[i + j] : 0.f;
    }
  };
  auto left4 = [&](int i, const float (&x)[4]) {         // which of them are left, a bit each
    unsigned b = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) b |= (unsigned)(i + j < s1 && ordered_key(x[j]) >= floor_key) << j;
    return b;
  };
  float sub = 0.f;
  for (int i0 = s0, it = 0; i0 < s1; i0 += blk, ++it) {
    float acc = 0.f;
    const int end = min(s1, i0 + blk);
    for (int i = i0; i < end; i += 512) {
      float x[4][4];
      unsigned left = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + 128 * u < end) values4(i + 128 * u + 4 * lane, x[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + 128 * u < end) left |= left4(i + 128 * u + 4 * lane, x[u]) << (4 * u);
      if (!__any_sync(0xffffffffu, left)) continue;      // (below a threshold most of a row is not left)
      auto add = [&](int u) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e = expf((x[u][j] - m) * invT);
          acc += left >> (4 * u + j) & 1u ? e : 0.f;
        }
      };
      add(0);
      if (i + 128 < end) { add(1); add(2); add(3); }     // (a short row's warps have 128 values)
    }
    acc = warp_sum(acc);
    if (lane == it) sub = acc;
  }
  float incl = sub;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (threadIdx.x == 0) found = -1;
  if (lane == 31) {
    if constexpr (BLOCKS == 2) pair_tell(scan + warp, incl);
    else scan[warp] = incl;
  }
  if constexpr (BLOCKS == 2) sc_barrier();
  else __syncthreads();
  if (threadIdx.x == 0) {
    float run = 0.f;
    const int nw = SAMPLE_THREADS >> 5;
    for (int w = 0; w < nw; ++w) { const float v = scan[w]; scan[w] = run; run += v; }
    scan[nw] = run;
  }
  __syncthreads();
  const float total = scan[SAMPLE_THREADS >> 5], all = __shfl_sync(0xffffffffu, incl, 31);
  const float before = scan[warp];
  const float u = uniform_draw(seeds ? seeds[r] : 0ULL, draw_index ? draw_index[r] : 0ULL);
  const float target = u * total;
  if (all > 0.f && target >= before && target < before + all) {
    const unsigned over = __ballot_sync(0xffffffffu, sub > 0.f && target < before + incl);
    // (rounding can leave none: then the last block with anything in it.  A lane's running sum starts from a sum in another
    // order than the one its neighbour ended with, so a draw can fall between the two: a value without weight, as a masked
    // one in a row without thresholds, is not taken for it)
    const unsigned some = __ballot_sync(0xffffffffu, sub > 0.f);
    const int b = over ? __ffs(over) - 1 : 31 - __clz(some);
    float cum = before + __shfl_sync(0xffffffffu, incl - sub, b);
    int pick = -1;
    const int i0 = s0 + b * blk, end = min(s1, i0 + blk);
    for (int i = i0; i < end; i += 128) {
      float x[4], w[4], sum = 0.f;
      const int at = i + 4 * lane;
      values4(at, x);
      const unsigned left = left4(at, x);
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = left >> j & 1u ? expf((x[j] - m) * invT) : -1.f;
      int last = -1;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (!(w[j] < 0.f)) sum += w[j];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (w[j] > 0.f) last = at + j;
      float run = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
      }
      float c = cum + (run - sum);
      int hit = -1;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (w[j] > 0.f) { c += w[j]; if (hit < 0 && target < c) hit = at + j; }
      const unsigned hits = __ballot_sync(0xffffffffu, hit >= 0), lasts = __ballot_sync(0xffffffffu, last >= 0);
      if (hits) { pick = __shfl_sync(0xffffffffu, hit, __ffs(hits) - 1); break; }
      if (lasts) pick = __shfl_sync(0xffffffffu, last, 31 - __clz(lasts));
      cum += __shfl_sync(0xffffffffu, run, 31);
    }
    if (lane == 0 && pick >= 0) atomicMax(&found, pick);
  }
  __syncthreads();
  if constexpr (BLOCKS == 2) {
    if (rank == 1 && threadIdx.x == 0) asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(pair_addr(&other_found)), "r"(found) : "memory");
    sc_barrier();
    if (tid == 0) found = max(found, other_found);
  }
  if (tid == 0) out[r] = found >= 0 ? found : amax;
}

// ---------------------------------------------------------------- a row on a cluster of CTAs
// One CTA per row reads its 128 k logits from L2 a dozen times (maximum, top-k and top-p
// descents of up to four passes each, sums), at the rate one SM gets from L2: 266 us with top-k
// and top-p before the descent was rewritten (43 us here, for 8 rows).  Here a row is cut into SC_CLUSTER parts, one per CTA of a cluster; a CTA reads
// its part from global memory once and keeps it in shared memory, and the CTAs exchange
// histograms and sums through distributed shared memory, always added in rank order, so every
// CTA takes the same decisions and the result is the same on every run.  Same arithmetic per
// element as sample_kernel; sums are associated differently (parts instead of 1024 strides).
#define SC_THREADS 512
#define SC_CLUSTER 8
#define SC_MIN_V 16384            // shorter rows stay with sample_kernel

// sum of v over the cluster in rank order (every CTA gets the same bits); *before = the sum
// over the ranks below this CTA's.  Called by all threads; v of thread 0 counts.
__device__ float sc_sum(float v, ClusterPub* pub, float* bcast, float* before) {
  const int par = pub->parity;
  if (threadIdx.x == 0) pub->f[par] = v;
  sc_barrier();
  if (threadIdx.x == 0) {
    const unsigned C = sc_size(), me = sc_rank();
    float run = 0.f, mine = 0.f;
    for (unsigned c = 0; c < C; ++c) {
      if (c == me) mine = run;
      run += sc_load(&pub->f[par], c);
    }
    bcast[0] = run;
    bcast[1] = mine;
    pub->parity = par ^ 1;
  }
  __syncthreads();
  if (before) *before = bcast[1];
  return bcast[0];
}

__global__ void __launch_bounds__(SC_THREADS)
sample_cluster_kernel(const float* __restrict__ logits, int V, int part, const float* __restrict__ temperature,
                      const int* __restrict__ top_k, const float* __restrict__ top_p,
                      const unsigned long long* __restrict__ seeds,
                      const unsigned long long* __restrict__ draw_index, int* __restrict__ out) {
  extern __shared__ __align__(16) float sc_part[];          // this CTA's part of the row
  __shared__ float red_f[33];
  __shared__ int red_i[33];
  __shared__ float hist[258];
  __shared__ __align__(8) unsigned bins[FX_PIECES * 256];
  __shared__ float scan[SC_THREADS / 32 + 1];
  __shared__ float bcast[2];
  __shared__ int found;
  __shared__ ClusterPub pub;
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.y;
  const unsigned me = sc_rank(), C = sc_size();
  const int base = (int)me * part, n = max(0, min(part, V - base));   // elements [base, base + n)
  const float* row = logits + (size_t)r * V;
  if (threadIdx.x == 0) pub.parity = 0;
  // the part into shared memory (float4 where the row's start allows it; part is a multiple of 4), its maximum on the way
  float best = -INFINITY;
  int bi = 0x7fffffff;
  auto seen = [&](float v, int i) { if (v > best) { best = v; bi = i; } };
  if (((((size_t)row) & 15) == 0) && (n & 3) == 0) {
    const float4* src = reinterpret_cast<const float4*>(row + base);
    float4* dst = reinterpret_cast<float4*>(sc_part);
#pragma unroll 4
    for (int i = threadIdx.x; i < (n >> 2); i += SC_THREADS) {
      const float4 v = src[i];
      dst[i] = v;
      seen(v.x, 4 * i); seen(v.y, 4 * i + 1); seen(v.z, 4 * i + 2); seen(v.w, 4 * i + 3);
    }
  } else {
    for (int i = threadIdx.x; i < n; i += SC_THREADS) { const float v = row[base + i]; sc_part[i] = v; seen(v, i); }
  }
  __syncthreads();
  const float T = temperature[r];
  // the maximum and its first index: of the part, then of the row (the lowest rank wins a tie)
  float m_local;
  const int a_local = first_if_none(first_of_block(best, bi, red_f, red_i, &m_local));
  if (threadIdx.x == 0) { pub.f[0] = n > 0 ? m_local : -INFINITY; pub.i[0] = base + a_local; }
  sc_barrier();
  float m = -INFINITY;
  int amax = 0;
  for (unsigned c = 0; c < C; ++c) {
    const float v = sc_load(&pub.f[0], c);
    if (v > m) { m = v; amax = sc_load(&pub.i[0], c); }
  }
  __syncthreads();
  if (threadIdx.x == 0) pub.parity = 1;
  __syncthreads();
  if (T <= 1e-9f) {
    if (me == 0 && threadIdx.x == 0) out[r] = amax;
    sc_barrier();                            // nobody leaves while a neighbour may still read it
    return;
  }
  const float invT = 1.f / T;
  unsigned int floor_key = 0;
  const int k = top_k ? top_k[r] : 0;
  if (k > 0 && k < V) floor_key = radix_threshold<false, 1>(sc_part, n, m, invT, 0u, (float)k, hist, red_f, bins, &pub);
  const float p = top_p ? top_p[r] : 0.f;
  if (p > 0.f && p < 1.f) {
    float z = 0.f;
    for (int i = threadIdx.x; i < n; i += SC_THREADS) {
      const float x = sc_part[i];
      if (ordered_key(x) >= floor_key) z += expf((x - m) * invT);
    }
    z = block_sum(z, red_f);
    z = sc_sum(z, &pub, bcast, nullptr);
    floor_key = radix_threshold<true, 1>(sc_part, n, m, invT, floor_key, p * z, hist, red_f, bins, &pub);
  }
  // running sum in index order over the kept elements: a thread owns a contiguous piece of
  // the part, a CTA the part, the ranks follow each other
  const int chunk = ((n + SC_THREADS - 1) / SC_THREADS) | 1;      // odd: the lanes' pieces start in different banks
  const int i0 = min(n, (int)threadIdx.x * chunk), i1 = min(n, i0 + chunk);
  float local = 0.f;
  for (int i = i0; i < i1; ++i) {
    const float x = sc_part[i];
    if (ordered_key(x) >= floor_key) local += expf((x - m) * invT);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (threadIdx.x == 0) found = -1;
  if (lane == 31) scan[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    float run = 0.f;
    for (int w = 0; w < SC_THREADS / 32; ++w) { const float v = scan[w]; scan[w] = run; run += v; }
    scan[SC_THREADS / 32] = run;
  }
  __syncthreads();
  float ranks_before;
  const float total = sc_sum(scan[SC_THREADS / 32], &pub, bcast, &ranks_before);
  const float before = ranks_before + scan[warp] + incl - local;
  const float u = uniform_draw(seeds ? seeds[r] : 0ULL, draw_index ? draw_index[r] : 0ULL);
  const float target = u * total;
  if (local > 0.f && target >= before && target < before + local) {
    float cum = before;
    int pick = -1;
    for (int i = i0; i < i1; ++i) {
      const float x = sc_part[i];
      if (ordered_key(x) >= floor_key) {
        const float w = expf((x - m) * invT);
        cum += w;
        if (w > 0.f) pick = base + i;            // (a draw that rounding carries past the end falls back to a value that can be drawn)
        if (target < cum) break;
      }
    }
    if (pick >= 0) atomicMax(&found, pick);
  }
  __syncthreads();
  // the largest index anybody found (rounding can make two neighbours claim the draw, or
  // nobody: then the maximum's index, as in sample_kernel)
  const int par = pub.parity;
  if (threadIdx.x == 0) pub.i[par] = found;
  sc_barrier();
  if (me == 0 && threadIdx.x == 0) {
    int best = -1;
    for (unsigned c = 0; c < C; ++c) best = max(best, sc_load(&pub.i[par], c));
    out[r] = best >= 0 ? best : amax;
  }
  sc_barrier();                              // nobody leaves while rank 0 may still read it
}

extern "C" int gg_argmax(const float* logits, int R, int V, int* out, cudaStream_t stream) {
  GG_REQUIRE(R >= 0 && V > 0, "argmax: bad sizes R=%d V=%d", R, V);
  if (R == 0) return GG_OK;
  gg_launch(argmax_kernel, dim3(R), dim3(SAMPLE_THREADS), 0, stream, logits, V, out);
  return gg_check_launch("argmax");
}

extern "C" int gg_sample(const float* logits, int R, int V, const float* temperature,
                         const int* top_k, const float* top_p, const unsigned long long* seeds,
                         const unsigned long long* draw_index, int* out, cudaStream_t stream) {
  GG_REQUIRE(R >= 0 && V > 0, "sample: bad sizes R=%d V=%d", R, V);
  GG_REQUIRE(temperature != nullptr, "sample: no temperatures given");
  if (R == 0) return GG_OK;
  static int use_cluster = -1;
  if (use_cluster < 0) { const char* e = getenv("GOLLMGO_B200_SAMPLE_CLUSTER"); use_cluster = e ? atoi(e) : 1; }
  const int part = (((V + SC_CLUSTER - 1) / SC_CLUSTER) + 3) & ~3;
  const size_t smem = (size_t)part * sizeof(float);
  static int num_sms = 0;
  if (!num_sms) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || num_sms <= 0)
      num_sms = 148;
  }
  // (with more rows than clusters fit at once, two CTAs per SM, two CTAs a row are faster: 37 rows of 128 k on clusters take 22 us
  // without thresholds, 46 with top-k, 70 with top-p alone, 38 rows in pairs 21, 32 and 58)
  if (use_cluster && V >= SC_MIN_V && smem <= 160 * 1024 && R * SC_CLUSTER <= 2 * num_sms) {
    static bool set = false;
    if (!set) {
      cudaError_t e = cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
      if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "sample: %s", cudaGetErrorString(e));
      set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SC_CLUSTER, R);
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SC_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gg_pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, sample_cluster_kernel, logits, V, part, temperature, top_k, top_p, seeds, draw_index, out);
    if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "sample: launch: %s", cudaGetErrorString(e));
    return gg_check_launch("sample");
  }
  // room for values in shared memory, most of a multiprocessor's: the registers of 1024 threads leave no second CTA anyway, and
  // how a row's sums are formed does not depend on how many rows there are (half of it for more rows than multiprocessors: 149
  // rows of 128 k with top_p alone 277 us against 189, flat ones 386 against 311; 200 with top_k as well 114 against 118)
  const int room = 48 * 1024, bytes = room * (int)sizeof(float);
  // two multiprocessors a row while there are two for each
  const bool pair = use_cluster && V >= SC_MIN_V && 2 * R <= num_sms;
  cudaError_t e = pair ? cudaFuncSetAttribute(sample_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)
                       : cudaFuncSetAttribute(sample_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "sample: %s", cudaGetErrorString(e));
  if (pair) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, R);
    cfg.blockDim = dim3(SAMPLE_THREADS / 2);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gg_pdl_enabled() ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, sample_kernel<2>, logits, V, temperature, top_k, top_p, seeds, draw_index, out, room);
    if (e != cudaSuccess) return gg_fail(GG_ERR_CUDA, "sample: launch: %s", cudaGetErrorString(e));
    return gg_check_launch("sample");
  }
  gg_launch(sample_kernel<1>, dim3(R), dim3(SAMPLE_THREADS), bytes, stream, logits, V, temperature, top_k, top_p, seeds, draw_index, out, room);
  return gg_check_launch("sample");
}
