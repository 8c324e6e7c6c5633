"""The plain linear recurrence S <- g S + k (beta v)^T, o = S^T q over a step's sequences, for the mixers built on it: prompt
portions in chunks as tensor-core products (csrc/linear_chunks.cu), short portions and single decoded tokens token by token
(csrc/delta_rule.cu)."""
from __future__ import annotations

import torch

from ..csrc import ops
from .context import QueryTiles

CHUNKS = QueryTiles(ops.LINEAR_CHUNK)
# Steps whose longest portion has so many tokens take the chunk form; below, its three kernels cost more than the walk (a B200,
# 64 heads of 64 with a state of 128, us for a layer, chunks and walk: one sequence of 128: 68 and 55, of 224: 75 and 76, of 256:
# 77 and 82, of 2048: 274 and 485; 32 of 128 after a context: 668 and 631, of 256: 1081 and 1226).
CHUNKS_FROM = 256


class PlainRecurrence:
    """Sizes: groups of q and k, heads, keys of d and values of dv.  ``chunks``: whether the chunk form may be used.  Its products
    of three tf32 parts and sums cut off at 24 bits are 1e-7 to 2e-6 from float64, the walk's 1e-7 to 4e-7: nothing beside the
    rounding of bfloat16 activations, but a model served in float32 keeps the walk."""

    def __init__(self, ctx, groups, heads, d, dv, chunks=True):
        self.ctx, self.sizes = ctx, (groups, heads, d, dv)
        self.chunked = chunks and ops.linear_chunks_ok(d, dv)
        if self.chunked:
            ctx.workspace.reserve("linear_states", ops.linear_scratch_floats(ctx.max_tokens, ctx.max_seqs, heads, d, dv), torch.float32)

    def query_tiles(self):
        return [CHUNKS] if self.chunked else []

    def run(self, rows, beta, decay, state, batch, out):
        groups, heads, d, dv = self.sizes
        seqs = (batch.cu_q_lens, batch.context_lens, batch.state_slots, batch.num_seqs)
        long = self.chunked and batch.num_portions and max(batch.q_lens) >= CHUNKS_FROM
        tiles = batch.tiles.get(CHUNKS) if long else None
        if tiles is not None:
            scratch = self.ctx.workspace.get("linear_states", 1, ops.linear_scratch_floats(out.shape[0], batch.num_seqs, heads, d, dv))
            if ops.linear_chunks(rows, beta, decay, state, scratch, tiles.seq, tiles.q0, tiles.count, *seqs, groups, heads, d, dv, out):
                if batch.num_decode:
                    ops.delta_recur(rows, beta, decay, state, *seqs, groups, heads, d, dv, out, plain=True, max_len=1)
                return
        ops.delta_recur(rows, beta, decay, state, *seqs, groups, heads, d, dv, out, plain=True)
