"""Steps of a gated delta rule layer that mix the chunk form, the walk and single tokens (parts/gated_delta.py): every sequence's state is
moved on once, whichever form takes it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D, H, G, DIM, TAPS, EPS = 64, 4, 2, 128, 4, 1e-5


class Layer:
    def __init__(self, weights, chunks, requests):
        from gollmgo_b200 import parts
        from gollmgo_b200.cache import CacheManager
        from gollmgo_b200.engine import BatchBuilder
        ctx = parts.BuildContext(torch.bfloat16, "cuda", max_tokens=2048, max_seqs=64, page_size=16)
        self.part = parts.build_mixer(parts.PartSpec("gated_delta", dict(hidden_size=D, num_heads=H, num_kv_heads=G, head_dim=DIM, v_head_dim=DIM,
                                                                         conv=TAPS, eps=EPS)), ctx)
        self.part.load(weights.__getitem__)
        if not chunks:
            self.part.chunks = None
        need = self.part.cache_need()
        self.cm = CacheManager([need], 16, 8, requests, dtype=torch.bfloat16, device="cuda")
        self.view = self.cm.cache_view(0, need)
        for t in self.view:
            t.zero_()
        for i in range(requests):
            self.cm.admit(i)
        self.builder = BatchBuilder(self.cm, "cuda", query_tiles=self.part.query_tiles())

    def step(self, x, lens):
        from gollmgo_b200.engine import StepEntry
        batch = self.builder.build([StepEntry(i, [0] * n, [0]) for i, n in enumerate(lens) if n])
        tiles = batch.tiles.get(self.part.chunks) if self.part.chunks is not None else None
        return self.part.forward(x, batch, self.view).clone(), tiles


@pytest.mark.parametrize("lens,listed,left_out", [
    ([600], 1, 0),                                         # nothing beside it
    ([513, 100, 1, 2], 3, 0),                              # short portions in chunks too, a single token
    ([512] + [9] * 40 + [1], 1, 40),                       # so many short ones that they are walked
    ([450, 1, 1, 700], 2, 0),                              # single tokens between long ones
])
def test_mixed_steps(lens, listed, left_out):
    from plain_bevuvik import gated_delta_rule
    gen = torch.Generator().manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=gen).bfloat16()  # noqa: E731
    kv, vv = G * DIM, H * DIM
    w = {"q": rnd(kv, D) / 8, "k": rnd(kv, D) / 8, "v": rnd(vv, D) / 8, "g": rnd(vv, D) / 8, "b": rnd(H, D) / 8, "a": rnd(H, D) / 8,
         "A_log": rnd(H) - 1.5, "dt_bias": rnd(H) / 2, "norm": 1 + rnd(DIM) / 5, "o": rnd(D, vv) / 16,
         "q.conv": rnd(kv, TAPS) / 2, "k.conv": rnd(kv, TAPS) / 2, "v.conv": rnd(vv, TAPS) / 2}
    on_gpu = {k: v.cuda() for k, v in w.items()}
    # five tokens each, the step in question on what they left, two single tokens on what it left
    steps = [[5] * len(lens), lens, [1] * len(lens), [1] * len(lens)]
    xs = [rnd(sum(s), D).cuda() for s in steps]
    layers = Layer(on_gpu, True, len(lens)), Layer(on_gpu, False, len(lens))
    rows = [[], []]
    for x, s in zip(xs, steps):
        for layer, out in zip(layers, rows):
            y, tiles = layer.step(x, s)
            out.append(y)
            if tiles is not None and s is lens:
                assert (tiles.left_out, len(set(tiles.seq.tolist()[:tiles.count]))) == (left_out, listed)
    torch.cuda.synchronize()
    # float32 sums in another order (4e-7 at most, test_delta_chunks.py); rows: roundings to bfloat16 that fall on the other side
    for a, b in zip(layers[0].view, layers[1].view):
        assert float((a - b).norm() / b.norm()) < 4e-6
    for a, b in zip(*rows):
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2e-3
    if len(lens) < 10:                                     # and the plain rule over the whole of the first and the last sequence
        for i in (0, len(lens) - 1):
            at = [sum(s[:i]) for s in steps]
            whole = torch.cat([x[a:a + s[i]] for x, a, s in zip(xs, at, steps)]).double().cpu()
            got = torch.cat([y[a:a + s[i]] for y, a, s in zip(rows[0], at, steps)]).double().cpu()
            want = gated_delta_rule(whole, {"p." + k: v.double() for k, v in w.items()}, "p.",
                                    dict(heads=H, kv_heads=G, dim=DIM, vdim=DIM, conv=TAPS), EPS)
            assert float((got - want).norm() / want.norm()) < 3e-2
