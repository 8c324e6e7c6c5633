"""The plain linear recurrence S <- g S + k (beta v)^T, o = S^T q over a step's sequences, for the mixers built on it: long prompt
portions in chunks as tensor-core products (csrc/linear_chunks.cu), short ones and single decoded tokens token by token
(csrc/delta_rule.cu).  A portion's own length decides, so its sums do not depend on what else is in the step."""
from __future__ import annotations

import torch

from ..csrc import ops
from .context import QueryTiles

# Portions of so many tokens take the chunk form: its three kernels, and the state that each chunk writes and reads, cost
# more than a shorter walk.  Steps of one portion, and of sixteen after a context (a B200, us for a layer, chunks / walk):
#   128 keys: 64 heads of 64      192: 74 / 70   256: 78 / 82    512: 111 / 140    16 x 256: 578 / 612   32 x 128: 678 / 616
#             128 heads of 64     192: 132 / 126 256: 142 / 146  512: 192 / 242    16 x 256: 1432 / 1477 32 x 128: 1673 / 1506
#             16 heads of 132     192: 69 / 60   256: 77 / 72    320: 82 / 86      16 x 256: 462 / 628   32 x 128: 496 / 630
#             32 heads of 132     192: 109 / 113 256: 119 / 131  512: 156 / 217    16 x 256: 1074 / 1414
#   64 keys:  64 heads of 64      256: 77 / 72   384: 93 / 93    512: 102 / 115    16 x 256: 502 / 464   8 x 512: 492 / 473
# (64 keys: the walk's cost goes with the keys, a chunk's with its rows.  A line at 512 there would leave the portions below it
# walking alone behind the chunks of a longer one: 364 + 218 + 582 + 436 tokens 296, all in chunks 231, all walking 328.)
def chunks_from(d):
    return 256 if d > 64 else 384


class PlainRecurrence:
    """Sizes: groups of q and k, heads, keys of d and values of dv.  ``chunks``: whether the chunk form may be used.  Its products
    of three tf32 parts and sums cut off at 24 bits are 1e-7 to 2e-6 from float64, the walk's 1e-7 to 4e-7: nothing beside the
    rounding of bfloat16 activations, but a model served in float32 keeps the walk."""

    def __init__(self, ctx, groups, heads, d, dv, chunks=True):
        self.ctx, self.sizes = ctx, (groups, heads, d, dv)
        self.limit = chunks_from(d)
        self.chunks = QueryTiles(ops.LINEAR_CHUNK, at_least=self.limit) if chunks and ops.linear_chunks_ok(d, dv) else None
        if self.chunks is not None:
            T = ctx.max_tokens
            ctx.workspace.reserve("linear_states", ops.linear_scratch_floats(T, T // self.limit, heads, d, dv), torch.float32)

    def query_tiles(self):
        return [self.chunks] if self.chunks is not None else []

    def run(self, rows, beta, decay, state, batch, out):
        groups, heads, d, dv = self.sizes
        seqs = (batch.cu_q_lens, batch.context_lens, batch.state_slots, batch.num_seqs)
        tiles = batch.tiles.get(self.chunks) if self.chunks is not None and batch.num_portions else None
        max_len = 0
        if tiles is not None and tiles.count:
            T = out.shape[0]
            scratch = self.ctx.workspace.get("linear_states", 1, ops.linear_scratch_floats(T, T // self.limit, heads, d, dv))
            if ops.linear_chunks(rows, beta, decay, state, scratch, tiles.seq, tiles.q0, tiles.count, *seqs, groups, heads, d, dv, out):
                if min(batch.q_lens) >= self.limit:
                    return
                max_len = self.limit - 1
        ops.delta_recur(rows, beta, decay, state, *seqs, groups, heads, d, dv, out, plain=True, max_len=max_len)
