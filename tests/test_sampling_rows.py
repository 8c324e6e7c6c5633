"""The sampling kernel with a row on one multiprocessor (csrc/sampling.cu): every way it finds its thresholds, against
probabilities in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from gollmgo_b200.csrc import ops
    return ops


def kept_probabilities(row, t, k, p):
    """Probabilities of the values that top-k and top-p leave (ties at a threshold all stay)."""
    x = row.double() / t
    if 0 < k < x.numel():
        x = x.masked_fill(x < x.topk(k).values[-1], -float("inf"))
    q = torch.softmax(x, 0)
    if 0 < p < 1:
        s, order = q.sort(descending=True)
        n = int((s.cumsum(0) < p - 1e-12).sum()) + 1
        q = torch.where(x >= x[order[n - 1]], q, torch.zeros_like(q))
        q = q / q.sum()
    return q


# vocabulary, rows, spread of the logits, (top_k, top_p) in turn: candidates above the threads' maxima; more than there are
# threads; a leading byte that fits in shared memory or does not (flat logits);
# odd widths (rows that start off a 16-byte border); fewer values than threads; rows whose integer sums need 64 bits
CASES = [(40000, 40, 2.5, [(50, 0.9), (1024, 0.0), (1025, 0.8), (3000, 0.95), (0, 0.9), (0, 0.0), (1, 0.5)]),
         (128256, 40, 2.5, [(0, 0.9), (400, 0.8), (0, 0.99), (20000, 0.5)]),
         (128256, 150, 0.4, [(0, 0.9), (400, 0.8), (0, 0.5)]),
         (60000, 40, 0.01, [(0, 0.9), (7, 0.9), (2000, 0.9)]),
         (16389, 60, 2.5, [(0, 0.9), (50, 0.0), (0, 0.0), (50, 0.7)]),
         (301, 5, 1.0, [(0, 0.9), (300, 0.7), (20, 0.0), (301, 0.4)]),
         (300000, 38, 1.5, [(0, 0.9), (100, 0.9), (5000, 0.6)])]


@pytest.mark.parametrize("V,R,std,ways", CASES)
def test_tokens_lie_where_the_draw_does(ops, V, R, std, ways):
    gen = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(R, V, device="cuda", generator=gen) * std
    logits[1] = torch.round(logits[1] * 4) / 4 + 0.0          # many ties (the kernels order -0 below 0, so there is none of it)
    logits[2, ::3] = -float("inf")
    dev = lambda x, dt: torch.tensor(x, dtype=dt, device="cuda")  # noqa: E731
    temps = [0.7 + 0.1 * (r % 4) for r in range(R)]
    ks, ps = [ways[r % len(ways)][0] for r in range(R)], [ways[r % len(ways)][1] for r in range(R)]
    args = (dev(temps, torch.float32), dev(ks, torch.int32), dev(ps, torch.float32), dev(list(range(R)), torch.int64), dev([3] * R, torch.int64))
    out, again = (torch.empty(R, dtype=torch.int32, device="cuda") for _ in range(2))
    ops.sample(logits, *args, out)
    ops.sample(logits, *args, again)
    assert torch.equal(out, again)
    mask = (1 << 64) - 1
    for r in range(R):
        z = (r + 4 * 0x9E3779B97F4A7C15) & mask
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        u = ((z ^ (z >> 31)) >> 40) / 2.0 ** 24
        q = kept_probabilities(logits[r], float(torch.tensor(temps[r], dtype=torch.float32)), ks[r], float(torch.tensor(ps[r], dtype=torch.float32)))
        cum, got = q.cumsum(0), int(out[r])
        # float32 sums of up to 3e5 weights: the draw may fall on a neighbour within 1e-4 of a border, and the nucleus may end a
        # value later or earlier, that is inside one of 1e-4 more
        p32 = float(torch.tensor(ps[r], dtype=torch.float32))
        wide = kept_probabilities(logits[r], float(torch.tensor(temps[r], dtype=torch.float32)), ks[r], p32 + 1e-4 if 0 < p32 < 1 else p32)
        assert wide[got] > 0, (r, got)
        assert float(cum[got] - q[got]) - 1e-4 <= u <= float(cum[got]) + 1e-4, (r, got)


@pytest.mark.parametrize("V", [16384, 40003, 128256, 262400])
@pytest.mark.parametrize("std", [2.5, 0.3])
def test_rows_on_two_multiprocessors_draw_what_they_draw_on_one(ops, V, std):
    """38 to 74 rows take two multiprocessors each, more of them one: the same sums in the same order, so the same tokens."""
    R, many = 64, 150
    gen = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(R, V, device="cuda", generator=gen) * std
    logits[1] = torch.round(logits[1] * 4) / 4 + 0.0
    logits[2, ::3] = -float("inf")
    logits[3, : V // 2] = logits[3, V // 2:V // 2 * 2]          # the maximum twice, in both halves of the threads
    logits[4, 7], logits[5, 9] = float("nan"), float("inf")
    logits[6] = -float("inf")
    ways = [(0, 0.9), (50, 0.9), (400, 0.0), (0, 0.0), (1024, 0.8), (3000, 0.95), (0, 0.3), (1, 0.0), (20000, 0.99)]
    for s in range(6):
        dev = lambda x, dt: torch.tensor(x, dtype=dt, device="cuda")  # noqa: E731
        args = (dev([0.0 if r % 11 == 3 else 0.6 + 0.1 * (r % 5) for r in range(many)], torch.float32),
                dev([ways[(r % R + s) % len(ways)][0] for r in range(many)], torch.int32),
                dev([ways[(r % R + s) % len(ways)][1] for r in range(many)], torch.float32),
                dev([r % R + 100 * s for r in range(many)], torch.int64), dev([3] * many, torch.int64))
        args = (args[0][torch.arange(many, device="cuda") % R].contiguous(), *args[1:])
        two, one = torch.empty(R, dtype=torch.int32, device="cuda"), torch.empty(many, dtype=torch.int32, device="cuda")
        ops.sample(logits, *(a[:R].contiguous() for a in args), two)
        ops.sample(logits[torch.arange(many, device="cuda") % R].contiguous(), *args, one)
        assert torch.equal(two, one[:R]) and torch.equal(one[R:2 * R], one[:R])
