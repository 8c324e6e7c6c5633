"""Which form of a linear recurrence a layer takes (parts/linear_recurrence.py, parts/retention.py)."""
import pytest
import torch

from gollmgo_b200.csrc import ops
from gollmgo_b200.parts import BuildContext, PartSpec, build_mixer

MIXERS = {
    "mamba2": dict(hidden_size=64, num_heads=4, v_head_dim=32, state=128, groups=2, conv=4, norm_groups=2, eps=1e-6),
    "mlstm": dict(hidden_size=64, num_heads=2, head_dim=128, v_head_dim=64, gate_cap=15.0, eps=1e-6),
    "retention": dict(hidden_size=64, num_heads=2, head_dim=128, v_head_dim=64, decay=[0.9, 0.99], eps=1e-6,
                      position=PartSpec("rope", dict(head_dim=128, theta=10000.0))),
}


def mixer(kind, dtype, device="cpu", max_tokens=2048, max_seqs=16):
    ctx = BuildContext(dtype, device, max_tokens=max_tokens, max_seqs=max_seqs, page_size=16)
    return build_mixer(PartSpec(kind, MIXERS[kind]), ctx), ctx


def chunk_lists(part):
    return [t for t in part.query_tiles() if t.height == ops.LINEAR_CHUNK]


@pytest.mark.parametrize("kind", sorted(MIXERS))
def test_models_in_float32_keep_float32_products(kind):
    assert chunk_lists(mixer(kind, torch.bfloat16)[0])
    assert not chunk_lists(mixer(kind, torch.float32)[0])


def listed(part, lens):
    """The sequences whose chunks a step of these portions lists, all of their chunks in order; and the portions it leaves out."""
    from gollmgo_b200.cache import CacheManager
    from gollmgo_b200.engine import BatchBuilder, StepEntry
    need, = chunk_lists(part)
    cm = CacheManager([part.cache_need()], 16, 8, len(lens), dtype=torch.bfloat16, device="cpu")
    for i in range(len(lens)):
        cm.admit(i)
    batch = BatchBuilder(cm, "cpu", query_tiles=part.query_tiles()).build([StepEntry(i, [0] * n, [0]) for i, n in enumerate(lens)])
    tiles = batch.tiles[need]
    seqs = sorted(set(tiles.seq.tolist()[:tiles.count]))
    assert list(zip(tiles.seq.tolist(), tiles.q0.tolist()))[:tiles.count] == [(b, q) for b in seqs for q in range(0, lens[b], ops.LINEAR_CHUNK)]
    assert tiles.left_out == sum(n > 1 for n in lens) - len(seqs)
    return seqs


@pytest.mark.parametrize("kind", sorted(MIXERS))
def test_long_portions_and_few_short_ones_beside_them(kind):
    part, _ = mixer(kind, torch.bfloat16, max_seqs=64)
    L = chunk_lists(part)[0].at_least
    assert listed(part, [L, 1, L - 1, 2, L + 129]) == [0, 2, 3, 4]                   # few chunks: the short ones beside the long
    assert listed(part, [L] + [8] * 40) == [0]                                       # many nearly empty ones: on their own
    assert listed(part, [1, L] + [100] * 9) == list(range(1, 11))                    # many well-filled ones
    assert listed(part, [L] + [40] * 9 + [L]) == [0, 10]
    assert listed(part, [1, 1]) == [] and listed(part, [20, 30, 1]) == []
    # portions that are only long together: retention alone
    assert listed(part, [L - 1, L - 1]) == ([0, 1] if kind == "retention" else [])
    assert listed(part, [16] * 20) == []


def test_keys_of_64_take_chunks_later():
    from gollmgo_b200.parts.linear_recurrence import PlainRecurrence
    need, = PlainRecurrence(BuildContext(torch.bfloat16, "cpu", max_tokens=4096, max_seqs=64, page_size=16), 1, 2, 64, 64).query_tiles()
    pick = lambda lens: need.chosen(list(range(len(lens))), lens, [0] * len(lens))  # noqa: E731
    assert pick([383]) == [] and pick([384]) == [0] and pick([256, 255]) == [] and pick([256, 256]) == [0, 1]
    assert pick([203, 121, 323]) == [0, 1, 2] and pick([256] * 16) == [] and pick([384] + [256] * 8) == list(range(9))


@pytest.mark.parametrize("kind", sorted(MIXERS))
def test_chunks_fit_in_the_scratch_whatever_the_step(kind):
    import random
    rng = random.Random(5)
    part, ctx = mixer(kind, torch.bfloat16, max_tokens=1024, max_seqs=64)
    need, = chunk_lists(part)
    name = "ret_states" if kind == "retention" else "linear_states"
    heads, d, dv = (part.nh, part.d, part.dv) if kind == "retention" else part.recurrence.sizes[1:]
    room = ctx.workspace._want[name][0] // (heads * (d * dv + 4))
    for _ in range(3000):
        lens, left = [], 1024
        while left > 1 and len(lens) < 64:
            n = min(left, rng.choice([2, 5, 20, 64, 65, 129, 130, 257, need.at_least, need.at_least + 1, rng.randint(2, 600)]))
            if n > 1:
                lens.append(n)
            left -= n
        chosen = need.chosen(list(range(len(lens))), lens, [0] * len(lens))
        assert sum(-(-lens[b] // ops.LINEAR_CHUNK) for b in chosen) <= room


@pytest.mark.parametrize("kind", ["mamba2", "mlstm"])
def test_scratch_is_for_chunks_of_long_portions(kind):
    """The states of the chunks that a step can hold, however many sequences a step may have."""
    few, many = (mixer(kind, torch.bfloat16, max_seqs=n)[1].workspace._want["linear_states"][0] for n in (1, 256))
    assert few == many
    part, ctx = mixer(kind, torch.bfloat16, max_tokens=4096)
    _, heads, d, dv = part.recurrence.sizes
    limit = part.recurrence.limit
    worst = max(n // p * -(-p // ops.LINEAR_CHUNK) for n in (4096,) for p in range(limit, 4097))
    assert worst <= ctx.workspace._want["linear_states"][0] // (heads * (d * dv + 4)) <= 4096 // 128 + 4096 // 256 + 1


@pytest.mark.gpu
@pytest.mark.parametrize("kind", sorted(MIXERS))
def test_long_short_and_single_portions_hand_one_state_on(kind):
    """The layer as it chooses beside the same layer without the chunk form, over steps that mix both with decoded tokens."""
    from gollmgo_b200 import parts
    from gollmgo_b200.cache import CacheManager
    from gollmgo_b200.engine import BatchBuilder, StepEntry
    parts.set_matmul_precision()
    # all in chunks; divided; single tokens; divided; all in chunks
    steps = [[300, 40, 1, 130, 1, 1, 1, 1], [300, 8, 8, 8, 8, 8, 8, 1], [1] * 8, [2, 600, 1, 20, 300, 2, 2, 2], [2, 255, 256, 1, 1, 1, 1, 1]]
    gen = torch.Generator(device="cuda").manual_seed(7)
    weights, sides, calls = {}, [], []
    for chunks in (True, False):
        part, ctx = mixer(kind, torch.bfloat16, "cuda")
        for n, s in part.weights().items():
            if n not in weights:
                w = torch.randn(*s.shape, device="cuda", generator=gen) * (s.shape[-1] ** -0.5 if len(s.shape) > 1 else 0.1)
                weights[n] = (w + (4.0 if n == "f.b" else -4.0 if n == "dt_bias" else 1.0 if n in ("norm", "D") else 0.0)).bfloat16()
        part.load(weights.__getitem__)
        if not chunks:
            if kind == "retention":
                part.tc = False
            else:
                part.recurrence.chunks = None
        cm = CacheManager([part.cache_need()], 16, 8, 8, dtype=torch.bfloat16, device="cuda")
        for i in range(8):
            cm.admit(i)
        view = cm.cache_view(0, part.cache_need())
        sides.append((part, BatchBuilder(cm, "cuda", query_tiles=part.query_tiles()), view))
    name = "linear_retention" if kind == "retention" else "linear_chunks"
    real = getattr(ops, name)
    for lens in steps:
        x = torch.randn(sum(lens), 64, device="cuda", generator=gen).bfloat16()
        got = []
        for part, builder, view in sides:
            setattr(ops, name, lambda *a, **k: calls.append(lens) or real(*a, **k))
            try:
                y = part.forward(x, builder.build([StepEntry(i, [0] * n, [0]) for i, n in enumerate(lens)]), view)
            finally:
                setattr(ops, name, real)
            got.append([y.float()] + [t.clone() for t in (view if isinstance(view, tuple) else (view,))])
        # what the rows' products differ by flips a bfloat16 rounding here and there (2^-9 of a value, for a few of the values);
        # the states are float32 on both sides, each within 4e-6 of float64
        assert float((got[0][0] - got[1][0]).norm() / got[1][0].norm()) < 2e-3
        for a, b in zip(got[0][1:], got[1][1:]):
            assert float((a.float() - b.float()).norm() / b.float().norm()) < 2e-5
    assert int(ops.tc_status("cuda")[0]) == 0
    assert calls == [lens for lens in steps if max(lens) > 255]
