// The short causal convolution + SiLU over time of the recurrent layers (delta_rule.cu, ssm.cu), four neighbouring
// channels a thread and several tokens one after another: the taps and the window stay in
// registers, and a row that four tokens use is read once and not four times.
// (Eight channels a thread are 16-byte loads, but 130 registers and a third of the warps: 27 us against 18 for the rows of
// a state-space layer of 4352 channels and 2048 tokens.)
#pragma once
#include "common.cuh"

#define CONV_THREADS 128
// Tokens of one block in a step with prompt portions: the rows before the block's first are read again (taps - 1 of them
// per CONV_TOKENS), fewer tokens a block would read more of them, more would leave multiprocessors without blocks.
#define CONV_TOKENS 16
// ... and fewer a block while there are no two blocks for every multiprocessor: a block walks its tokens one after another.  Us for
// a layer on a B200 with 16 / 4 / 1 tokens a block: state space (6144 channels), six prompts of 34 tokens together 49 / 43 / 43,
// one of 200 78 / 74 / 76, of 512 120 / 119 / 127, of 2048 288 / 291 / 326; delta rule (3072), 34: 46 / 39 / 38, 83 + 50 + 132 + 99
// 100 / 92 / 95, 512: 141 / 135 / 138, 2048: 473 / 477 / 489.
inline int conv_tokens_a_block(int T, int B, int groups) {
  if (T <= 4 * B) return 1;
  int per = CONV_TOKENS;
  while (per > 1 && (long long)((T + per - 1) / per) * groups < 2 * 148) per /= 2;
  return per;
}

// Index of the sequence that token t belongs to: the largest b with cu[b] <= t.
__device__ __forceinline__ int seq_of_token(const int* __restrict__ cu, int B, int t) {
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Channels c .. c + 3 of tokens [ta, tb) of x (rows of x_stride values, whose channel 0 is x[0]); emit(t, y) gets the
// four results of token t: all threads of a warp call it together for the same t, since the lanes of a head sum among
// themselves, so threads without channels of their own (live = false) go the same way and only store nothing.  conv_state
// [slots, TAPS - 1, C] holds the inputs before each sequence's first token of the step.  `single` (as many tokens as sequences, [ta, tb) one token): the
// thread that reads a sequence's window is the only one that does, so it also moves the window on.
template <int TAPS, typename TA, typename Emit>
__device__ __forceinline__ void conv_tokens(const TA* __restrict__ x, long long x_stride, const float* __restrict__ conv_w,
                                            const float* __restrict__ conv_b, float* conv_state,
                                            const int* __restrict__ cu, const int* __restrict__ context_lens,
                                            const int* __restrict__ state_slots, int B, int C, int c, int ta, int tb,
                                            bool single, bool live, Emit emit) {
  float w[TAPS * 4];
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f), win[TAPS - 1];
#pragma unroll
  for (int i = 0; i < TAPS; ++i) {
    const float4 v = *reinterpret_cast<const float4*>(conv_w + (size_t)c * TAPS + 4 * i);
    w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
  }
  if (conv_b) bias = load4(conv_b + c);
  pdl_wait();
  const TA* xc = x + c;
  int b = seq_of_token(cu, B, ta);
  tb = min(tb, cu[B]);                                 // (rows behind the last sequence have no window)
  for (int t = ta; t < tb; ++b) {
    const int t0 = cu[b], t1 = cu[b + 1], slot = state_slots[b];
    const bool carried = slot >= 0 && context_lens[b] - (t1 - t0) > 0;
    float* st = conv_state + (size_t)(carried ? slot : 0) * (TAPS - 1) * C + c;
#pragma unroll
    for (int s = 0; s < TAPS - 1; ++s) {
      const int src = t - t0 - (TAPS - 1) + s;
      if (src >= 0) win[s] = load4(xc + (size_t)(t0 + src) * x_stride);
      else if (carried) win[s] = load4(st + (size_t)(TAPS - 1 + src) * C);
      else win[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (single && t != t0) return;                       // (a sequence of several tokens all the same: its first block takes them)
    const int te = single ? t1 : min(tb, t1);
    while (t < te) {
      float4 row[4];                                     // four rows on their way before the first is used
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (t + k < te) row[k] = load4(xc + (size_t)(t + k) * x_stride);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (t + k >= te) break;
        float4 acc = bias;
#pragma unroll
        for (int s = 0; s < TAPS; ++s) {
          const float4 v = s < TAPS - 1 ? win[s] : row[k];
          acc.x = fmaf(w[s], v.x, acc.x);
          acc.y = fmaf(w[TAPS + s], v.y, acc.y);
          acc.z = fmaf(w[2 * TAPS + s], v.z, acc.z);
          acc.w = fmaf(w[3 * TAPS + s], v.w, acc.w);
        }
#pragma unroll
        for (int s = 0; s + 1 < TAPS - 1; ++s) win[s] = win[s + 1];
        win[TAPS - 2] = row[k];
        float4 y = make_float4(acc.x / (1.f + expf(-acc.x)), acc.y / (1.f + expf(-acc.y)), acc.z / (1.f + expf(-acc.z)), acc.w / (1.f + expf(-acc.w)));
        emit(t + k, y);
      }
      t = min(te, t + 4);
    }
    if (single && live && slot >= 0) {
      float* to = conv_state + (size_t)slot * (TAPS - 1) * C + c;
#pragma unroll
      for (int s = 0; s < TAPS - 1; ++s) store4(to + (size_t)s * C, win[s]);
    }
  }
}
