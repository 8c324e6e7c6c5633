"""Which portions of a gated delta rule layer take the chunk form (parts/gated_delta.py)."""
import pytest
import torch

from gollmgo_b200.csrc import ops
from gollmgo_b200.parts import BuildContext, PartSpec, build_mixer


def mixer(dtype=torch.bfloat16, d=128, dv=128, decay="head", max_tokens=2048):
    ctx = BuildContext(dtype, "cpu", max_tokens=max_tokens, max_seqs=64, page_size=16)
    return build_mixer(PartSpec("gated_delta", dict(hidden_size=64, num_heads=2, num_kv_heads=1, head_dim=d, v_head_dim=dv, conv=4,
                                                    eps=1e-6, decay=decay)), ctx)


def test_forms_that_keep_the_walk():
    assert mixer().query_tiles()
    assert not mixer(torch.float32).query_tiles() and not mixer(decay="channel").query_tiles()
    assert not mixer(d=48).query_tiles() and not mixer(dv=24).query_tiles() and not mixer(d=256).query_tiles()


@pytest.mark.parametrize("d", [64, 128])
def test_long_portions_and_few_short_ones_beside_them(d):
    from gollmgo_b200.cache import CacheManager
    from gollmgo_b200.engine import BatchBuilder, StepEntry
    part = mixer(d=d)
    need, = part.query_tiles()
    L = need.at_least
    for lens, want in (([L, 1, L - 1, 2], [0, 2, 3]), ([L] + [8] * 40, [0]), ([L - 1, L - 1], []), ([1, 1], []), ([3 * L], [0])):
        cm = CacheManager([part.cache_need()], 16, 8, len(lens), dtype=torch.bfloat16, device="cpu")
        for i in range(len(lens)):
            cm.admit(i)
        tiles = BatchBuilder(cm, "cpu", query_tiles=[need]).build([StepEntry(i, [0] * n, [0]) for i, n in enumerate(lens)]).tiles[need]
        listed = list(zip(tiles.seq.tolist(), tiles.q0.tolist()))[:tiles.count]
        assert listed == [(b, q) for b in want for q in range(0, lens[b], ops.LINEAR_CHUNK)]
        # what the scratch is made for
        assert part.scratch[0] >= tiles.count * 2 * (d * 128 + 4)
        assert part.scratch[1] >= tiles.count * 128 * 3 * d + sum(lens) * 2


def test_scratch_holds_the_most_tiles():
    part = mixer(max_tokens=1000)
    need, = part.query_tiles()
    assert part.scratch[0] >= need.most * 2 * (128 * 128 + 4) and part.scratch[1] >= need.most * 128 * 3 * 128 + 1000 * 2
