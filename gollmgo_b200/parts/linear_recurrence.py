"""The plain linear recurrence S <- g S + k (beta v)^T, o = S^T q over a step's sequences, for the mixers built on it: long prompt
portions in chunks as tensor-core products (csrc/linear_chunks.cu), short ones and single decoded tokens token by token
(csrc/delta_rule.cu)."""
from __future__ import annotations

from dataclasses import dataclass

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
# (64 keys: the walk's cost goes with the keys, a chunk's with its rows.)
def chunks_from(d):
    return 256 if d > 64 else 384


@dataclass(frozen=True)
class ChunkTiles(QueryTiles):
    """The chunks of a step: of the portions of ``at_least`` rows; but of all portions, the short ones too, where the longest has
    ``longest`` rows, all together ``rows``, and the chunks are few or filled well, at most ``most``.  The two forms of a step
    run one after the other and the walk is as long as its longest portion, so a few short portions are cheaper beside the
    long ones' chunks, many nearly empty chunks dearer (a B200, us for a layer, portions after a context; all in chunks /
    divided): retention 16 heads 128 x 256, 108 + 65 + 171 + 128 + 85: 102 / 169; state space 64 heads, 128 keys, 235 + 141 +
    375 + 281 + 187 + 421: 250 / 314, 2048 + 15 x 128: 589 / 563, 300 + 63 x 8: 782 / 253; 16 heads of 132, 1024 + 4 x 100:
    188 / 201, 2048 + 15 x 128: 471 / 539, 300 + 63 x 8: 408 / 202."""
    longest: int = 0
    rows: int = 0
    most: int = 0

    __hash__ = QueryTiles.__hash__

    def chosen(self, portions, q_lens, q_starts):
        lens = [q_lens[b] for b in portions]
        total = sum(lens)
        longest = max(lens, default=0)
        if total >= self.rows and longest >= self.longest:
            tiles = sum(-(-n // self.height) for n in lens)
            if tiles <= self.most and (tiles <= FEW_CHUNKS or (longest >= self.at_least and total >= FILLED * tiles)):
                return portions
        return super().chosen(portions, q_lens, q_starts)


# Few chunks fit on the machine together (64 heads of a group: sixteen blocks a chunk); of more, each has to have so many of its
# 128 tokens (retention 16 heads 128 x 256 after a context, all in chunks / packed float32: 8 x 64: 95 / 121, 32 x 64: 444 / 366,
# 20 x 192: 541 / 582, 32 x 16: 300 / 204).
FEW_CHUNKS, FILLED = 8, 80


class PlainRecurrence:
    """Sizes: groups of q and k, heads, keys of d and values of dv.  ``chunks``: whether the chunk form may be used.  Its products
    of three tf32 parts and sums cut off at 24 bits are 1e-7 to 2e-6 from float64, the walk's 1e-7 to 4e-7: nothing beside the
    rounding of bfloat16 activations, but a model served in float32 keeps the walk."""

    def __init__(self, ctx, groups, heads, d, dv, chunks=True):
        self.ctx, self.sizes = ctx, (groups, heads, d, dv)
        self.limit, self.chunks = chunks_from(d), None
        if chunks and ops.linear_chunks_ok(d, dv):
            T = ctx.max_tokens
            # (64 keys: 203 + 121 + 323 tokens all in chunks 128 us, walked 133; 16 x 256 divided by the line above)
            self.chunks = ChunkTiles(ops.LINEAR_CHUNK, at_least=self.limit, longest=256, rows=0 if d > 64 else 512,
                                     most=T // ops.LINEAR_CHUNK + T // self.limit)
            ctx.workspace.reserve("linear_states", ops.linear_scratch_floats(T, T // self.limit, heads, d, dv), torch.float32)

    def query_tiles(self):
        return [self.chunks] if self.chunks is not None else []

    def run(self, rows, beta, decay, state, batch, out):
        groups, heads, d, dv = self.sizes
        tiles, max_len = batch.tiles.get(self.chunks), 0
        if tiles is not None and tiles.count:
            T = self.ctx.max_tokens
            scratch = self.ctx.workspace.get("linear_states", 1, ops.linear_scratch_floats(T, T // self.limit, heads, d, dv))
            if ops.linear_chunks(rows, beta, decay, state, scratch, tiles.seq, tiles.q0, tiles.count, batch.cu_q_lens, batch.context_lens,
                                 batch.state_slots, batch.num_seqs, groups, heads, d, dv, out):
                if not tiles.left_out and not batch.num_decode:
                    return
                max_len = self.limit - 1 if tiles.left_out else 1
        ops.delta_recur(rows, beta, decay, state, batch.cu_q_lens, batch.context_lens, batch.state_slots, batch.num_seqs, groups, heads,
                        d, dv, out, True, max_len)
