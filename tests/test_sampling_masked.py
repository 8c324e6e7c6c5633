"""What a draw may return (csrc/sampling.cu): a value without weight never, a value outside top-k or the nucleus neither; many draws
a row, since a wrong pick sits in the rounding between two lanes' sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def draw(logits, temps, ks, ps, seeds):
    from gollmgo_b200.csrc import ops
    R = logits.shape[0]
    dev = lambda x, dt: torch.as_tensor(x, dtype=dt).to("cuda")  # noqa: E731
    out = torch.empty(R, dtype=torch.int32, device="cuda")
    ops.sample(logits, dev(temps, torch.float32), dev(ks, torch.int32), dev(ps, torch.float32), dev(seeds, torch.int64),
               dev([5] * R, torch.int64), out)
    return out.long()


# rows on clusters of eight multiprocessors, and a row a multiprocessor
@pytest.mark.parametrize("V,R", [(128256, 148), (128256, 16), (4099, 148)])
def test_masked_values_are_never_drawn(V, R):
    gen = torch.Generator(device="cuda").manual_seed(V + R)
    drawn = 0
    for k in range(20):
        logits = torch.randn(R, V, device="cuda", generator=gen) * 2.5
        logits[:, k % 3::3] = -float("inf")
        for s in range(25):
            got = draw(logits, [1.0] * R, [0] * R, [0.0] * R, [(k * 25 + s) * R + r for r in range(R)])
            assert bool(torch.isfinite(logits.gather(1, got[:, None])).all()), (k, s)
            drawn += R
    assert drawn == 500 * R                                # (148 rows of 128 k: one in ten thousand was wrong before)


@pytest.mark.parametrize("V,R,std", [(128256, 148, 2.5), (128256, 30, 2.5), (40000, 148, 0.3), (515, 40, 1.0)])
def test_draws_stay_inside_top_k_and_the_nucleus(V, R, std):
    gen = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(R, V, device="cuda", generator=gen) * std
    logits[:, ::3] = -float("inf")
    ways = [(0, 0.9), (50, 0.0), (50, 0.8), (1, 0.9), (400, 0.95), (0, 0.3), (1500, 0.5)]
    ks, ps = [ways[r % len(ways)][0] for r in range(R)], [ways[r % len(ways)][1] for r in range(R)]
    lowest = torch.empty(R, dtype=torch.float64, device="cuda")
    for r in range(R):
        x = logits[r].double()
        if 0 < ks[r] < V:
            x = x.masked_fill(x < x.topk(ks[r]).values[-1], -float("inf"))
        if ps[r] > 0:
            # the threshold of a nucleus of 1e-4 more: what float32 sums of up to V weights can be off by
            s, order = torch.softmax(x, 0).sort(descending=True)
            n = min(int((s.cumsum(0) < float(torch.tensor(ps[r])) + 1e-4).sum()) + 1, int((s > 0).sum()))
            lowest[r] = x[order[n - 1]]
        else:
            lowest[r] = x[torch.isfinite(x)].min()
    for s in range(60):
        got = draw(logits, [1.0] * R, ks, ps, [1000 * s + r for r in range(R)])
        value = logits.gather(1, got[:, None])[:, 0].double()
        assert bool((torch.isfinite(value) & (value >= lowest)).all()), s
