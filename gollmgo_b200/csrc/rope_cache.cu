// Rotary position encoding of q and k, fused with the write of k and v into the
// paged cache.
//
// Reference: kernels/gollmgo_ops.cu:321-358 (rope, adjacent pairs, theta fixed at
// 10000) followed by kernels/gollmgo_paged_attn.cu:126-146 (scatter by slot).  Here
// the inverse frequencies come from a table the host builds from config.json
// (theta, rope_scaling), the pairing is half-split (p, p+rot/2) unless
// `interleaved`, and one kernel does both so k and v are read once.
//
// qkv:   [T, (nh + 2*nkv) * d]   q heads, then k heads, then v heads; q and k are
//        rotated in place (k also lands rotated in the cache)
// cache: K and V of one layer, each [num_pages, nkv, page_size, d]
// slot:  slot_mapping[t] = page * page_size + offset, or < 0 to skip the write
// inv_freq: rot/2 doubles, or null for no rotation (then only the cache write happens)
// The angle pos * inv_freq is formed and reduced modulo 2 pi in float64; sine, cosine
// and the rotation itself are float32.
#include "common.cuh"

#define ROPE_HEADS_PER_CTA 8

// grid (T, ceil((nh + 2 nkv) / 8)): a CTA takes eight consecutive heads (q, k or v) of one token.
template <typename TA>
__global__ void rope_kv_write_kernel(TA* __restrict__ qkv, const int* __restrict__ positions,
                                     const int* __restrict__ slot_mapping,
                                     const double* __restrict__ inv_freq, TA* __restrict__ kcache,
                                     TA* __restrict__ vcache, int nh, int nkv, int d, int rot,
                                     int page_size, int interleaved, int write_cache) {
  extern __shared__ float cs[];        // cos[rot/2], sin[rot/2]
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  const int half = rot >> 1;
  const int h0 = blockIdx.y * ROPE_HEADS_PER_CTA;
  const int h1 = min(h0 + ROPE_HEADS_PER_CTA, nh + 2 * nkv);
  const bool rotates = inv_freq && h0 < nh + nkv;
  if (rotates) {
    // angle in float64, reduced to [-pi, pi] in float64, then float32 sine and cosine: the
    // reduction keeps the accuracy of the float64 product at any position, and the float32
    // functions are exact to an ulp on the reduced argument
    const double pos = (double)positions[t];
    const double two_pi = 6.283185307179586476925286766559;
    for (int p = threadIdx.x; p < half; p += blockDim.x) {
      const double ang = pos * inv_freq[p];
      const float r = (float)(ang - two_pi * rint(ang * (1.0 / two_pi)));
      float s, c;
      sincosf(r, &s, &c);
      cs[p] = c;
      cs[half + p] = s;
    }
  }
  __syncthreads();
  const int slot = (write_cache && slot_mapping) ? slot_mapping[t] : -1;
  const int page = slot >= 0 ? slot / page_size : 0;
  const int off = slot >= 0 ? slot - page * page_size : 0;
  TA* row = qkv + (size_t)t * (nh + 2 * nkv) * d;

  for (int h = h0; h < h1; ++h) {
    TA* x = row + (size_t)h * d;
    if (h < nh + nkv) {
      // a q or k head: rotate `half` pairs, copy the rest of a k head to the cache as it is
      TA* kc = (h >= nh && slot >= 0) ? kcache + (((size_t)page * nkv + (h - nh)) * page_size + off) * d : nullptr;
      if (inv_freq) {
        for (int p = threadIdx.x; p < half; p += blockDim.x) {
          const int i0 = interleaved ? 2 * p : p;
          const int i1 = interleaved ? 2 * p + 1 : p + half;
          const float a = to_f32(x[i0]), b = to_f32(x[i1]);
          const float c = cs[p], s = cs[half + p];
          const TA ra = from_f32<TA>(a * c - b * s);
          const TA rb = from_f32<TA>(a * s + b * c);
          x[i0] = ra;
          x[i1] = rb;
          if (kc) { kc[i0] = ra; kc[i1] = rb; }
        }
      }
      if (kc) {
        const int from = inv_freq ? rot : 0;
        for (int c = from + threadIdx.x; c < d; c += blockDim.x) kc[c] = x[c];
      }
    } else if (slot >= 0) {
      TA* vcp = vcache + (((size_t)page * nkv + (h - nh - nkv)) * page_size + off) * d;
      for (int c = threadIdx.x; c < d; c += blockDim.x) vcp[c] = x[c];
    }
  }
}

// The common case at full width: bfloat16, half-split pairs, the whole head rotated, head size a
// multiple of 16.  One CTA per token; a thread takes eight pairs of one head with two 16-byte
// loads (columns p..p+7 and p+d/2..p+d/2+7), or eight values of a v head, and stores in kind.
__global__ void __launch_bounds__(256)
rope_kv_write_vec_kernel(__nv_bfloat16* __restrict__ qkv, const int* __restrict__ positions,
                         const int* __restrict__ slot_mapping, const double* __restrict__ inv_freq,
                         __nv_bfloat16* __restrict__ kcache, __nv_bfloat16* __restrict__ vcache, int nh, int nkv,
                         int d, int page_size, int write_cache) {
  extern __shared__ float cs[];        // cos[d/2], sin[d/2]
  pdl_trigger();
  const int t = blockIdx.x;
  const int half = d >> 1;
  // The token's position and cache slot were copied in before the step began and the
  // frequencies never change: the table of cosines and sines is ready before the kernel
  // ahead (the qkv product) has finished; only the rows of qkv have to wait for it.
  {
    const double pos = (double)positions[t];
    const double two_pi = 6.283185307179586476925286766559;
    for (int p = threadIdx.x; p < half; p += blockDim.x) {
      const double ang = pos * inv_freq[p];
      const float r = (float)(ang - two_pi * rint(ang * (1.0 / two_pi)));
      float s, c;
      sincosf(r, &s, &c);
      cs[p] = c;
      cs[half + p] = s;
    }
  }
  const int slot = (write_cache && slot_mapping) ? slot_mapping[t] : -1;
  __syncthreads();
  pdl_wait();
  const int page = slot >= 0 ? slot / page_size : 0;
  const int off = slot >= 0 ? slot - page * page_size : 0;
  __nv_bfloat16* row = qkv + (size_t)t * (nh + 2 * nkv) * d;
  const int per_head = half >> 3;                       // groups of eight pairs per head
  const int rot_items = (nh + nkv) * per_head, v_items = nkv * (d >> 3);
  for (int e = threadIdx.x; e < rot_items + v_items; e += blockDim.x) {
    if (e < rot_items) {
      const int h = e / per_head, p0 = (e - h * per_head) << 3;
      __nv_bfloat16* x = row + (size_t)h * d;
      uint4 lo = *reinterpret_cast<const uint4*>(x + p0), hi = *reinterpret_cast<const uint4*>(x + half + p0);
      __nv_bfloat162* a2 = reinterpret_cast<__nv_bfloat162*>(&lo);
      __nv_bfloat162* b2 = reinterpret_cast<__nv_bfloat162*>(&hi);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(a2[i]), b = __bfloat1622float2(b2[i]);
        const float c0 = cs[p0 + 2 * i], s0 = cs[half + p0 + 2 * i], c1 = cs[p0 + 2 * i + 1], s1 = cs[half + p0 + 2 * i + 1];
        a2[i] = __floats2bfloat162_rn(a.x * c0 - b.x * s0, a.y * c1 - b.y * s1);
        b2[i] = __floats2bfloat162_rn(a.x * s0 + b.x * c0, a.y * s1 + b.y * c1);
      }
      *reinterpret_cast<uint4*>(x + p0) = lo;
      *reinterpret_cast<uint4*>(x + half + p0) = hi;
      if (h >= nh && slot >= 0) {
        __nv_bfloat16* kc = kcache + (((size_t)page * nkv + (h - nh)) * page_size + off) * d;
        *reinterpret_cast<uint4*>(kc + p0) = lo;
        *reinterpret_cast<uint4*>(kc + half + p0) = hi;
      }
    } else if (slot >= 0) {
      const int ev = e - rot_items;
      const int h = ev / (d >> 3), c = (ev - h * (d >> 3)) << 3;
      *reinterpret_cast<uint4*>(vcache + (((size_t)page * nkv + h) * page_size + off) * d + c) =
          *reinterpret_cast<const uint4*>(row + (size_t)(nh + nkv + h) * d + c);
    }
  }
}

extern "C" int gg_rope_kv_write(void* qkv, int act_dtype, const int* positions,
                                const int* slot_mapping, const double* inv_freq, void* kcache,
                                void* vcache, int T, int nh, int nkv, int d, int rot,
                                int page_size, int interleaved, int write_cache,
                                cudaStream_t stream) {
  GG_REQUIRE(T >= 0 && nh > 0 && nkv > 0 && d > 0 && page_size > 0,
             "rope_kv_write: bad sizes T=%d nh=%d nkv=%d d=%d page=%d", T, nh, nkv, d, page_size);
  GG_REQUIRE(rot >= 0 && rot <= d && rot % 2 == 0, "rope_kv_write: rotary width %d must be even and <= head size %d", rot, d);
  GG_REQUIRE(!write_cache || (kcache && vcache && slot_mapping), "rope_kv_write: cache write without cache or slots");
  if (T == 0) return GG_OK;
  if (rot == 0) inv_freq = nullptr;
  const size_t smem = (size_t)rot * sizeof(float);
  GG_REQUIRE(smem <= 48 * 1024, "rope_kv_write: rotary width %d too large", rot);
  if (act_dtype == GG_BF16 && inv_freq && rot == d && d % 16 == 0 && !interleaved &&
      ((size_t)qkv % 16) == 0 && (!write_cache || (((size_t)kcache % 16) == 0 && ((size_t)vcache % 16) == 0))) {
    gg_launch(rope_kv_write_vec_kernel, dim3(T), dim3(256), smem, stream, (__nv_bfloat16*)qkv, positions, slot_mapping,
              inv_freq, (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, nh, nkv, d, page_size, write_cache);
    return gg_check_launch("rope_kv_write");
  }
  const int threads = d >= 256 ? 128 : 64;
  const dim3 grid(T, (nh + 2 * nkv + ROPE_HEADS_PER_CTA - 1) / ROPE_HEADS_PER_CTA);
  GG_REQUIRE(grid.y <= 65535, "rope_kv_write: too many heads");
  if (act_dtype == GG_F32)
    gg_launch(rope_kv_write_kernel<float>, grid, dim3(threads), smem, stream, (float*)qkv, positions, slot_mapping, inv_freq, (float*)kcache, (float*)vcache, nh, nkv, d, rot, page_size, interleaved, write_cache);
  else if (act_dtype == GG_BF16)
    gg_launch(rope_kv_write_kernel<__nv_bfloat16>, grid, dim3(threads), smem, stream, (__nv_bfloat16*)qkv, positions, slot_mapping, inv_freq, (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, nh, nkv, d, rot, page_size, interleaved, write_cache);
  else
    return gg_fail(GG_ERR_INVALID, "rope_kv_write: unknown dtype %d", act_dtype);
  return gg_check_launch("rope_kv_write");
}

// The same for projections of any make: key heads of size d and value heads of size dv in
// numbers of their own, an optional bias on the whole row (added first, in float32), rotation
// of the first `rot` values of every q and k head, and a factor `mag` on every cosine and sine
// (rotary tables that are stretched for long contexts scale both).
// row:   [nh*d | nkv*d | nv*dv]
// cache: K [num_pages, nkv, page_size, d], V [num_pages, nv, page_size, dv]
template <typename TA>
__global__ void rope_kv_write_x_kernel(TA* __restrict__ qkv, long long row_stride, const int* __restrict__ positions,
                                       const int* __restrict__ slot_mapping, const double* __restrict__ inv_freq,
                                       float mag, const float* __restrict__ bias, TA* __restrict__ kcache,
                                       TA* __restrict__ vcache, int nh, int nkv, int d, int nv, int dv, int rot,
                                       int page_size, int interleaved, int write_cache) {
  extern __shared__ float cs[];        // cos[rot/2], sin[rot/2]
  pdl_trigger();
  const int t = blockIdx.x;
  const int half = rot >> 1;
  const int h0 = blockIdx.y * ROPE_HEADS_PER_CTA;
  const int h1 = min(h0 + ROPE_HEADS_PER_CTA, nh + nkv + nv);
  if (inv_freq && h0 < nh + nkv) {
    const double pos = (double)positions[t];
    const double two_pi = 6.283185307179586476925286766559;
    for (int p = threadIdx.x; p < half; p += blockDim.x) {
      const double ang = pos * inv_freq[p];
      const float r = (float)(ang - two_pi * rint(ang * (1.0 / two_pi)));
      float s, c;
      sincosf(r, &s, &c);
      cs[p] = c * mag;
      cs[half + p] = s * mag;
    }
  }
  const int slot = (write_cache && slot_mapping) ? slot_mapping[t] : -1;
  __syncthreads();
  pdl_wait();
  const int page = slot >= 0 ? slot / page_size : 0;
  const int off = slot >= 0 ? slot - page * page_size : 0;
  TA* row = qkv + (size_t)t * row_stride;
  for (int h = h0; h < h1; ++h) {
    if (h < nh + nkv) {
      TA* x = row + (size_t)h * d;
      const float* b = bias ? bias + (size_t)h * d : nullptr;
      TA* kc = (h >= nh && slot >= 0) ? kcache + (((size_t)page * nkv + (h - nh)) * page_size + off) * d : nullptr;
      const int nrot = inv_freq ? half : 0;
      for (int p = threadIdx.x; p < nrot; p += blockDim.x) {
        const int i0 = interleaved ? 2 * p : p;
        const int i1 = interleaved ? 2 * p + 1 : p + half;
        const float u = to_f32(x[i0]) + (b ? b[i0] : 0.f), v = to_f32(x[i1]) + (b ? b[i1] : 0.f);
        const float c = cs[p], s = cs[half + p];
        const TA ru = from_f32<TA>(u * c - v * s);
        const TA rv = from_f32<TA>(v * c + u * s);
        x[i0] = ru;
        x[i1] = rv;
        if (kc) { kc[i0] = ru; kc[i1] = rv; }
      }
      for (int c = 2 * nrot + threadIdx.x; c < d; c += blockDim.x) {
        const TA y = b ? from_f32<TA>(to_f32(x[c]) + b[c]) : x[c];
        if (b) x[c] = y;
        if (kc) kc[c] = y;
      }
    } else {
      const int hv = h - nh - nkv;
      TA* x = row + (size_t)(nh + nkv) * d + (size_t)hv * dv;
      const float* b = bias ? bias + (size_t)(nh + nkv) * d + (size_t)hv * dv : nullptr;
      TA* vcp = slot >= 0 ? vcache + (((size_t)page * nv + hv) * page_size + off) * dv : nullptr;
      if (!b && !vcp) continue;
      for (int c = threadIdx.x; c < dv; c += blockDim.x) {
        const TA y = b ? from_f32<TA>(to_f32(x[c]) + b[c]) : x[c];
        if (b) x[c] = y;
        if (vcp) vcp[c] = y;
      }
    }
  }
}

// The common case of it: bfloat16, half-split pairs, sizes and starts in groups of eight values.  One CTA per token; a
// thread takes eight pairs (two 16-byte loads), or eight values that pass, and stores in kind.  2048 tokens of 32 + 2 x 8
// heads of 128 without a rotation: 6.5 us (a value at a time: 24).
__global__ void __launch_bounds__(256)
rope_kv_write_x_vec_kernel(__nv_bfloat16* __restrict__ qkv, long long row_stride, const int* __restrict__ positions,
                           const int* __restrict__ slot_mapping, const double* __restrict__ inv_freq, float mag,
                           const float* __restrict__ bias, __nv_bfloat16* __restrict__ kcache, __nv_bfloat16* __restrict__ vcache, int nh,
                           int nkv, int d, int nv, int dv, int rot, int page_size, int write_cache) {
  extern __shared__ float cs[];        // cos[rot/2], sin[rot/2]
  pdl_trigger();
  const int t = blockIdx.x;
  const int half = rot >> 1;
  if (half) {
    const double pos = (double)positions[t];
    const double two_pi = 6.283185307179586476925286766559;
    for (int p = threadIdx.x; p < half; p += blockDim.x) {
      const double ang = pos * inv_freq[p];
      const float r = (float)(ang - two_pi * rint(ang * (1.0 / two_pi)));
      float s, c;
      sincosf(r, &s, &c);
      cs[p] = c * mag;
      cs[half + p] = s * mag;
    }
  }
  const int slot = (write_cache && slot_mapping) ? slot_mapping[t] : -1;
  __syncthreads();
  pdl_wait();
  const int page = slot >= 0 ? slot / page_size : 0;
  const int off = slot >= 0 ? slot - page * page_size : 0;
  __nv_bfloat16* row = qkv + (size_t)t * row_stride;
  const int per_rot = half >> 3, per_pass = (d - rot) >> 3, per_v = dv >> 3;
  const int h_pass = bias ? 0 : nh;                      // without a bias a q head's values that pass stay as they are
  const int n_rot = (nh + nkv) * per_rot, n_pass = (nh + nkv - h_pass) * per_pass, n_v = nv * per_v;
  auto add8 = [&](uint4& r, const float* b) {
    __nv_bfloat162* a = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(a[i]);
      a[i] = __floats2bfloat162_rn(f.x + b[2 * i], f.y + b[2 * i + 1]);
    }
  };
  for (int e = threadIdx.x; e < n_rot + n_pass + n_v; e += blockDim.x) {
    if (e < n_rot) {
      const int h = e / per_rot, p0 = (e - h * per_rot) << 3;
      __nv_bfloat16* x = row + (size_t)h * d;
      uint4 lo = *reinterpret_cast<const uint4*>(x + p0), hi = *reinterpret_cast<const uint4*>(x + half + p0);
      __nv_bfloat162* a2 = reinterpret_cast<__nv_bfloat162*>(&lo);
      __nv_bfloat162* b2 = reinterpret_cast<__nv_bfloat162*>(&hi);
      const float* bl = bias ? bias + (size_t)h * d + p0 : nullptr;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 a = __bfloat1622float2(a2[i]), b = __bfloat1622float2(b2[i]);
        if (bl) { a.x += bl[2 * i]; a.y += bl[2 * i + 1]; b.x += bl[half + 2 * i]; b.y += bl[half + 2 * i + 1]; }
        const float c0 = cs[p0 + 2 * i], s0 = cs[half + p0 + 2 * i], c1 = cs[p0 + 2 * i + 1], s1 = cs[half + p0 + 2 * i + 1];
        a2[i] = __floats2bfloat162_rn(a.x * c0 - b.x * s0, a.y * c1 - b.y * s1);
        b2[i] = __floats2bfloat162_rn(b.x * c0 + a.x * s0, b.y * c1 + a.y * s1);
      }
      *reinterpret_cast<uint4*>(x + p0) = lo;
      *reinterpret_cast<uint4*>(x + half + p0) = hi;
      if (h >= nh && slot >= 0) {
        __nv_bfloat16* kc = kcache + (((size_t)page * nkv + (h - nh)) * page_size + off) * d;
        *reinterpret_cast<uint4*>(kc + p0) = lo;
        *reinterpret_cast<uint4*>(kc + half + p0) = hi;
      }
    } else {
      const bool is_v = e >= n_rot + n_pass;
      const int i = e - n_rot - (is_v ? n_pass : 0), per = is_v ? per_v : per_pass;
      const int hh = i / per, h = is_v ? hh : h_pass + hh, c = (is_v ? 0 : rot) + ((i - hh * per) << 3);
      const size_t at = (is_v ? (size_t)(nh + nkv) * d + (size_t)h * dv : (size_t)h * d) + c;
      __nv_bfloat16* to = nullptr;
      if (slot >= 0 && is_v) to = vcache + (((size_t)page * nv + h) * page_size + off) * dv + c;
      else if (slot >= 0 && h >= nh) to = kcache + (((size_t)page * nkv + (h - nh)) * page_size + off) * d + c;
      if (!bias && !to) continue;
      uint4 v = *reinterpret_cast<const uint4*>(row + at);
      if (bias) {
        add8(v, bias + at);
        *reinterpret_cast<uint4*>(row + at) = v;
      }
      if (to) *reinterpret_cast<uint4*>(to) = v;
    }
  }
}

extern "C" int gg_rope_kv_write_x(void* qkv, long long row_stride, int act_dtype, const int* positions,
                                  const int* slot_mapping, const double* inv_freq, float mag, const float* bias,
                                  void* kcache, void* vcache, int T, int nh, int nkv, int d, int nv, int dv, int rot,
                                  int page_size, int interleaved, int write_cache, cudaStream_t stream) {
  // nv = 0: the rows hold no values of their own (a layer whose values are its keys)
  GG_REQUIRE(T >= 0 && nh > 0 && nkv > 0 && d > 0 && nv >= 0 && dv > 0 && page_size > 0,
             "rope_kv_write_x: bad sizes T=%d nh=%d nkv=%d d=%d nv=%d dv=%d page=%d", T, nh, nkv, d, nv, dv, page_size);
  GG_REQUIRE(rot >= 0 && rot <= d && rot % 2 == 0, "rope_kv_write_x: rotary width %d must be even and <= head size %d", rot, d);
  GG_REQUIRE(row_stride >= (long long)(nh + nkv) * d + (long long)nv * dv, "rope_kv_write_x: rows of %lld values are too short", row_stride);
  GG_REQUIRE(!write_cache || (kcache && vcache && slot_mapping), "rope_kv_write_x: cache write without cache or slots");
  if (T == 0) return GG_OK;
  const size_t smem = (size_t)(rot > 0 ? rot : 2) * sizeof(float);
  GG_REQUIRE(smem <= 48 * 1024, "rope_kv_write_x: rotary width %d too large", rot);
  if (!inv_freq) rot = 0;                                // without a table every value passes
  if (rot == 0) inv_freq = nullptr;
  if (act_dtype == GG_BF16 && !(interleaved && rot) && d % 8 == 0 && dv % 8 == 0 && rot % 16 == 0 && row_stride % 8 == 0 && ((size_t)qkv % 16) == 0 &&
      (!write_cache || (((size_t)kcache % 16) == 0 && ((size_t)vcache % 16) == 0))) {
    gg_launch(rope_kv_write_x_vec_kernel, dim3(T), dim3(256), smem, stream, (__nv_bfloat16*)qkv, row_stride, positions, slot_mapping,
              inv_freq, mag, bias, (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, nh, nkv, d, nv, dv, rot, page_size, write_cache);
    return gg_check_launch("rope_kv_write_x");
  }
  const int big = d > dv ? d : dv;
  const int threads = big >= 256 ? 128 : 64;
  const dim3 grid(T, (nh + nkv + nv + ROPE_HEADS_PER_CTA - 1) / ROPE_HEADS_PER_CTA);
  GG_REQUIRE(grid.y <= 65535, "rope_kv_write_x: too many heads");
  if (act_dtype == GG_F32)
    gg_launch(rope_kv_write_x_kernel<float>, grid, dim3(threads), smem, stream, (float*)qkv, row_stride, positions, slot_mapping, inv_freq, mag, bias, (float*)kcache, (float*)vcache, nh, nkv, d, nv, dv, rot, page_size, interleaved, write_cache);
  else if (act_dtype == GG_BF16)
    gg_launch(rope_kv_write_x_kernel<__nv_bfloat16>, grid, dim3(threads), smem, stream, (__nv_bfloat16*)qkv, row_stride, positions, slot_mapping, inv_freq, mag, bias, (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache, nh, nkv, d, nv, dv, rot, page_size, interleaved, write_cache);
  else
    return gg_fail(GG_ERR_INVALID, "rope_kv_write_x: unknown dtype %d", act_dtype);
  return gg_check_launch("rope_kv_write_x");
}
