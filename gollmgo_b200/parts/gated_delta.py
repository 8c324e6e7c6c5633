"""The gated delta rule: a recurrent mixer whose state per head is a matrix S [d, dv],

    S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q,

with q and k (``num_kv_heads`` heads of size ``head_dim``, shared by ``num_heads / num_kv_heads``
value heads each) and v (``num_heads`` heads of size ``v_head_dim``) passed through a short causal
convolution and SiLU, q and k made unit vectors (q times head_dim^-1/2), beta = sigmoid(Wb x),
g = exp(-exp(A_log) * softplus(Wa x + dt_bias)) per head.  The result is divided by its root mean
square per head, multiplied by a weight shared by the heads and by silu(Wg x), and projected.

State per request, in its state slot: S in float32 [heads, dv, d] and the last taps - 1 inputs
of the convolution in float32 [taps - 1, channels].  Nothing is paged.  Everything between the
projections and the output projection is float32 (csrc/delta_rule.cu; long prompt portions with a decay per
head in chunks, csrc/delta_chunks.cu).

Variants, all parameters: ``decay="channel"``: g is a factor per head and key channel (a row of S,
``dt_bias`` then [heads * head_dim]) instead of one per head; ``a_rank`` / ``gate_rank``: the
decay's input and the output gate come through two products of that inner width (tensors a1, a2 and
g1, g2) instead of one; ``gate_act="sigmoid"``: the output gate is a sigmoid instead of SiLU.

params: hidden_size, num_heads, num_kv_heads, head_dim, v_head_dim, conv (taps), eps, out_buffer,
decay ("head" | "channel"), a_rank, gate_rank (None: one product; else the inner width that random
weights are made with: a checkpoint's tensors decide), gate_act ("silu" | "sigmoid"),
names (optional dict: q, k, v, beta, a, gate, o, A_log, dt_bias, norm, a1, a2, g1, g2; the
convolutions' tensors are the q, k, v names + ".conv").
"""
from __future__ import annotations

import math
from dataclasses import dataclass

import torch

from ..cache import FixedStateNeed
from ..csrc import ops
from ..weights import WeightSpec
from .linear import linear, linear_with_tail
from .linear_recurrence import ChunkTiles
from .registry import register_mixer

# Portions of so many tokens may take the chunk form (csrc/delta_chunks.cu).  A B200, us, chunks / walk, values of 128, 16 heads on 4
# (128 keys also 32 on 8):
#   128 keys: 256: 56 / 50, 67 / 64   320: 64 / 62, 82 / 80   384: 68 / 74, 88 / 95   512: 76 / 97, 98 / 126   2048: 212 / 382, 336 / 497
#   64 keys:  256: 41 / 37            384: 49 / 55            512: 52 / 73            2048: 133 / 284
CHUNKS_FROM = 384


@dataclass(frozen=True)
class DeltaTiles(ChunkTiles):
    """ChunkTiles for steps whose chunks are also estimated to take less time than the walk.  The walk takes its longest portion's
    tokens one after the other until its blocks, sixteen value columns of a sequence and head each, fill the machine, and then what all
    of them take; the chunks their fixed cost, one chunk after the other, and the arithmetic of all.  Estimates in us, each of two
    parts as the root of their squares' sum; of 165 steps measured on a B200 (11 kinds of layer, 1 to 20 portions of 64 to 2048 tokens)
    117 and 142 took what is estimated to within a tenth, and none in chunks took over 1 % longer than walked.  What decides between them, chunks / walk: 16 heads, 64 keys, 8 x 384 tokens: 179 / 157, one of 384:
    49 / 55; 48 heads of 64 x 64, 700 + 513 + 835: 259 / 196, one of 2048: 261 / 337; 4 heads of 32 x 16, 20 x 512: 100 / 69."""
    heads: int = 1
    d: int = 128
    dv: int = 128

    __hash__ = ChunkTiles.__hash__

    def chunk_us(self, lens):
        D, cols = (64 if self.d <= 64 else 128), (64 if self.dv <= 64 else -(-self.dv // 128) * 128)       # (as the kernels pad them)
        chunks = [-(-n // 64) for n in lens]
        return (30 if cols <= 128 else 40) + math.hypot((0.06 + 1.5e-5 * D * cols) * self.heads * sum(chunks), 0.027 * D * max(chunks))

    def walk_us(self, lens):
        return math.hypot((0.095 + 7.2e-4 * self.d) * max(lens), (1.3e-4 + 4.2e-6 * self.d) * sum(lens) * self.heads * self.dv / 16)

    def chosen(self, portions, q_lens, q_starts):
        listed = super().chosen(portions, q_lens, q_starts)
        if not listed:
            return listed
        here = set(listed)
        rest = [q_lens[b] for b in portions if b not in here]          # walked behind the chunks
        cost = self.chunk_us([q_lens[b] for b in listed]) + (5 + self.walk_us(rest) if rest else 0)
        return listed if 1.04 * cost < self.walk_us([q_lens[b] for b in portions]) else []


def one_kernel(B, groups, heads, d, dv):
    """Whether B single tokens go through delta_step (csrc/delta_rule.cu) and not through three kernels.  It saves two launches, but has a
    block of 512 threads a sequence and head, and clusters of the heads that share q and k.  A B200, us with a small product behind, one
    kernel / three, 64 x 64: 4 heads, 1: 4.8 / 7.4; 48 heads on 6 (clusters of eight), 8: 10.9 / 12.6, 16: 17.6 / 16.5; 32 on 8, 32: 15.9 /
    15.7, 64: 30.5 / 24.5.  128 x 128: 16 on 4, 8: 8.1 / 12.9, 32: 20.3 / 22.4; 8 on 1, 16: 11.5 / 12.6, 32: 14.4 / 13.9.  64 x 128:
    48 on 6, 16: 25.0 / 25.6.  64 x 256: 16 on
    4, 16: 17.3 / 20.1, 32: 25.3 / 24.3; 8 on 1, 8: 9.0 / 10.6, 16: 14.6 / 13.9.  128 x 256, half the state in registers: 8 heads, 4: 11.1
    / 10.3, 8: 11.1 / 13.4.  (And no more than 32 MB of states: the kernel's own limit.)"""
    blocks = B * heads
    if dv == 256:
        return (48 if d == 128 else 1) <= blocks <= (64 if heads == 8 * groups else 256)
    if heads == 8 * groups:
        return blocks <= (768 if d != dv else 512 if d == 64 else 192)
    return blocks <= 1024


_NAMES = {"q": "q", "k": "k", "v": "v", "beta": "b", "a": "a", "gate": "g", "o": "o", "A_log": "A_log",
          "dt_bias": "dt_bias", "norm": "norm", "a1": "a1", "a2": "a2", "g1": "g1", "g2": "g2"}


class GatedDeltaRule:
    def __init__(self, spec, ctx):
        self.ctx = ctx
        self.hidden = int(spec["hidden_size"])
        self.nh = int(spec["num_heads"])
        self.nkv = int(spec["num_kv_heads"])
        self.d = int(spec["head_dim"])
        self.dv = int(spec["v_head_dim"])
        self.taps = int(spec["conv"])
        self.eps = float(spec["eps"])
        self.names = dict(_NAMES, **(spec.get("names") or {}))
        self.out_buffer = spec.get("out_buffer") or "mixer_out"
        if self.nh % self.nkv:
            raise ValueError(f"{self.nh} heads are not a multiple of {self.nkv} q/k heads")
        if self.d > 256:
            raise ValueError(f"key size {self.d} is beyond what the recurrence kernel takes (256)")
        if not (1 <= self.taps <= 17):
            raise ValueError(f"{self.taps} taps are outside 1..17")
        decay = spec.get("decay") or "head"
        if decay not in ("head", "channel"):
            raise ValueError(f"decay {decay!r} is not known (known: head, channel)")
        self.dw = self.d if decay == "channel" else 1                        # decays per head and token
        self.a_rank = int(spec.get("a_rank") or 0)
        self.gate_rank = int(spec.get("gate_rank") or 0)
        self.gate_act = spec.get("gate_act") or "silu"
        if self.gate_act not in ("silu", "sigmoid"):
            raise ValueError(f"gate activation {self.gate_act!r} is not known (known: silu, sigmoid)")
        self.channels = 2 * self.nkv * self.d + self.nh * self.dv            # q, k, v: what the convolution sees
        self._layout()
        ws, T = ctx.workspace, ctx.max_tokens
        ws.reserve("delta_ba", T * self.nh * (1 + self.dw), torch.float32)
        ws.reserve("delta_qkv", T * self.channels, torch.float32)
        ws.reserve("delta_beta", T * self.nh, torch.float32)
        ws.reserve("delta_decay", T * self.nh * self.dw, torch.float32)
        if self.gate_rank:
            ws.reserve("delta_gate", T * self.nh * self.dv, ctx.act_dtype)
        ws.reserve("delta_o", T * self.nh * self.dv, torch.float32)
        ws.reserve("delta_y", T * self.nh * self.dv, ctx.act_dtype)
        ws.reserve(self.out_buffer, T * self.hidden, ctx.act_dtype)
        # (float32 arithmetic too, its sums in another order: a model served in float32 keeps the walk's)
        self.chunks = None
        if self.dw == 1 and ctx.act_dtype != torch.float32 and ops.delta_chunks_ok(self.d, self.dv):
            limit = CHUNKS_FROM
            self.chunks = DeltaTiles(ops.LINEAR_CHUNK, at_least=limit, longest=limit, most=T // ops.LINEAR_CHUNK + T // limit,
                                     heads=self.nh, d=self.d, dv=self.dv)
            self.scratch = (ops.linear_scratch_floats(T, T // limit, self.nh, self.d, self.dv),
                            ops.delta_solved_floats(T, T // limit, self.nkv, self.nh, self.d, self.dv))
            ws.reserve("linear_states", self.scratch[0], torch.float32)
            ws.reserve("delta_solved", self.scratch[1], torch.float32)
        self.w_all = self.w_proj = self.w_ba = self.w_o = self.w_a2 = self.w_g2 = None
        self.conv_w = self.a_log = self.dt_bias = self.norm_w = None

    def _layout(self):
        """Columns of the stacked first product: q, k, v, then the gate (or its inner values), then the
        decay's inner values; every part starts at a multiple of 8 columns."""
        pad8 = lambda n: -(-n // 8) * 8
        self.gate_col = pad8(self.channels)
        self.gate_cols = self.gate_rank or self.nh * self.dv
        self.a_col = pad8(self.gate_col + self.gate_cols)
        self.proj_width = pad8(self.a_col + self.a_rank) if self.a_rank else pad8(self.gate_col + self.gate_cols)
        self.ctx.workspace.reserve("delta_proj", self.ctx.max_tokens * self.proj_width, self.ctx.act_dtype)

    def cache_need(self):
        need = [FixedStateNeed((self.nh, self.dv, self.d), "float32")]
        if self.taps > 1:
            need.append(FixedStateNeed((self.taps - 1, self.channels), "float32"))
        return tuple(need)

    def weights(self):
        n = self.names
        qk, vv = self.nkv * self.d, self.nh * self.dv
        w = {n["q"]: WeightSpec((qk, self.hidden)), n["k"]: WeightSpec((qk, self.hidden)),
             n["v"]: WeightSpec((vv, self.hidden)),
             n["beta"]: WeightSpec((self.nh, self.hidden)),
             n["A_log"]: WeightSpec((self.nh,), init="normal"),
             n["dt_bias"]: WeightSpec((self.nh * self.dw,), init="normal"),
             n["norm"]: WeightSpec((self.dv,)), n["o"]: WeightSpec((self.hidden, vv))}
        if self.gate_rank:
            # the inner widths are the checkpoint's: what the parameters say is what random weights are made with
            w[n["g1"]] = WeightSpec((self.gate_rank, self.hidden), free_dims=(0,))
            w[n["g2"]] = WeightSpec((vv, self.gate_rank), free_dims=(1,))
        else:
            w[n["gate"]] = WeightSpec((vv, self.hidden))
        if self.a_rank:
            w[n["a1"]] = WeightSpec((self.a_rank, self.hidden), free_dims=(0,))
            w[n["a2"]] = WeightSpec((self.nh * self.dw, self.a_rank), free_dims=(1,))
        else:
            w[n["a"]] = WeightSpec((self.nh * self.dw, self.hidden))
        w.update({n["q"] + ".conv": WeightSpec((qk, self.taps), init="taps"),
                  n["k"] + ".conv": WeightSpec((qk, self.taps), init="taps"),
                  n["v"] + ".conv": WeightSpec((vv, self.taps), init="taps")})
        return w

    def load(self, get):
        n = self.names
        parts = [get(n[x]) for x in ("q", "k", "v")] + [get(n["g1"] if self.gate_rank else n["gate"])]
        if self.a_rank:
            parts.append(get(n["a1"]))
        ranks = (parts[3].shape[0] if self.gate_rank else 0, parts[4].shape[0] if self.a_rank else 0)
        if self.gate_rank and get(n["g2"]).shape[1] != ranks[0] or self.a_rank and get(n["a2"]).shape[1] != ranks[1]:
            raise ValueError("the two products of a low-rank input disagree in their inner width")
        if ranks != (self.gate_rank, self.a_rank):
            self.gate_rank, self.a_rank = ranks
            self._layout()
        dt = torch.float32 if any(p.dtype == torch.float32 for p in parts) else parts[0].dtype
        w_proj = torch.zeros(self.proj_width, self.hidden, dtype=dt, device=parts[0].device)
        w_proj[:self.channels] = torch.cat([p.to(dt) for p in parts[:3]], dim=0)
        w_proj[self.gate_col:self.gate_col + self.gate_cols] = parts[3].to(dt)
        if self.a_rank:
            w_proj[self.a_col:self.a_col + self.a_rank] = parts[4].to(dt)
            # the decay's second product reads the padded inner values: columns of zeros for the padding
            a2 = get(n["a2"])
            self.w_a2 = torch.zeros(a2.shape[0], self.proj_width - self.a_col, dtype=a2.dtype, device=a2.device)
            self.w_a2[:, :self.a_rank] = a2
            self.w_ba = get(n["beta"]).contiguous()
        else:
            self.w_ba = torch.cat([get(n["beta"]), get(n["a"])], dim=0).contiguous()
        if self.gate_rank:
            g2 = get(n["g2"])
            self.w_g2 = torch.zeros(g2.shape[0], self.a_col - self.gate_col if self.a_rank else self.proj_width - self.gate_col,
                                    dtype=g2.dtype, device=g2.device)
            self.w_g2[:, :self.gate_rank] = g2
        self.w_all, self.w_proj = None, w_proj.contiguous()
        if self.w_ba.dtype == dt == torch.bfloat16:        # one behind the other: steps of a few tokens multiply both in one launch
            self.w_all = torch.cat([self.w_proj, self.w_ba], dim=0)
            self.w_proj, self.w_ba = self.w_all[:self.proj_width], self.w_all[self.proj_width:]
        self.w_o = get(n["o"]).contiguous()
        self.conv_w = torch.cat([get(n[x] + ".conv").float() for x in ("q", "k", "v")], dim=0).contiguous()
        self.a_log = get(n["A_log"]).float().contiguous()
        self.dt_bias = get(n["dt_bias"]).float().contiguous()
        self.norm_w = get(n["norm"]).float().contiguous()

    def query_tiles(self):
        return [self.chunks] if self.chunks is not None else []

    def _recur(self, qkv, beta, decay, state, batch, o):
        B, H, d, dv = batch.num_seqs, self.nh, self.d, self.dv
        tiles, max_len = batch.tiles.get(self.chunks) if self.chunks is not None else None, 0
        if tiles is not None and tiles.count:
            states, solved = (self.ctx.workspace.get(n, 1, size) for n, size in zip(("linear_states", "delta_solved"), self.scratch))
            if ops.delta_chunks(qkv, beta, decay, state, states, solved, tiles.seq, tiles.q0, tiles.count, batch.cu_q_lens,
                                batch.context_lens, batch.state_slots, B, self.nkv, H, d, dv, o):
                if not tiles.left_out and not batch.num_decode:
                    return
                max_len = self.chunks.at_least - 1 if tiles.left_out else 1
        ops.delta_recur(qkv, beta, decay, state, batch.cu_q_lens, batch.context_lens, batch.state_slots, B, self.nkv, H, d, dv, o,
                        max_len=max_len)

    def forward(self, x, batch, cache, writes_cache=True, then=None):
        T = x.shape[0]
        ws = self.ctx.workspace
        state = cache[0]
        conv_state = cache[1] if self.taps > 1 else state        # unused without taps to carry
        H, hw = self.nh, self.nh * self.dw
        proj, ba = ws.get("delta_proj", T, self.proj_width), ws.get("delta_ba", T, H + hw)
        if self.a_rank:
            # beta straight from x; the decay's input through its two products (the inner values are columns of proj)
            proj, zb = linear_with_tail(x, self.w_all, self.w_proj, self.w_ba, proj, ba.view(-1)[:T * H].view(T, H))
            za = linear(proj[:, self.a_col:], self.w_a2, ba.view(-1)[T * H:].view(T, hw))
        else:
            proj, ba = linear_with_tail(x, self.w_all, self.w_proj, self.w_ba, proj, ba)
            zb, za = ba[:, :H], ba[:, H:]
        y = ws.get("delta_y", T, self.nh * self.dv)
        if self.gate_rank:
            gate = linear(proj[:, self.gate_col:self.a_col if self.a_rank else self.proj_width], self.w_g2,
                          ws.get("delta_gate", T, self.nh * self.dv))
        else:
            gate = proj[:, self.gate_col:self.gate_col + self.gate_cols]
        B = batch.num_seqs
        if T == B and batch.num_portions == 0 and self.dw == 1 and self.taps > 1 and proj.dtype == torch.bfloat16 \
                and one_kernel(B, self.nkv, H, self.d, self.dv) and ops.delta_step(
                    proj, self.conv_w, conv_state, zb, za, self.a_log, self.dt_bias, state, batch.cu_q_lens, batch.context_lens,
                    batch.state_slots, B, self.nkv, H, self.d, self.dv, gate, self.norm_w, self.eps, y, self.gate_act):
            return linear(y, self.w_o, ws.get(self.out_buffer, T, self.hidden), then)
        qkv = ws.get("delta_qkv", T, self.channels)
        beta, decay = ws.get("delta_beta", T, H), ws.get("delta_decay", T, hw)
        ops.delta_prep(proj, self.conv_w, conv_state, zb, za, self.a_log, self.dt_bias, batch.cu_q_lens, batch.context_lens,
                       batch.state_slots, B, self.nkv, self.nh, self.d, self.dv, qkv, beta, decay)
        o = ws.get("delta_o", T, self.nh * self.dv)
        self._recur(qkv, beta, decay, state, batch, o)
        ops.delta_out(o, gate, self.norm_w, self.eps, self.nh, self.dv, y, self.gate_act)
        return linear(y, self.w_o, ws.get(self.out_buffer, T, self.hidden), then)


register_mixer("gated_delta", GatedDeltaRule)
