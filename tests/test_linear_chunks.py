"""The plain linear recurrence in chunks (csrc/linear_chunks.cu) against float64 and beside the token-by-token kernel: chunks of
128 tokens at their edges, carried states, single tokens left alone, decays from none to total; and retention on the same kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from gollmgo_b200.csrc import ops
    return ops


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def walk(q, k, v, decay, beta, S):
    """Token by token in float64: q, k [T, H, d], v [T, H, dv], decay and beta [T, H], S [H, dv, d]."""
    out = torch.empty_like(v)
    for t in range(v.shape[0]):
        S = S * decay[t][:, None, None] + (beta[t][:, None] * v[t])[:, :, None] * k[t][:, None, :]
        out[t] = (S * q[t][:, None, :]).sum(-1)
    return out, S


@pytest.mark.parametrize("G,H,d,dv", [(1, 8, 128, 64), (2, 4, 64, 128), (3, 3, 128, 132), (2, 2, 8, 4), (1, 2, 256, 256), (2, 2, 72, 200)])
@pytest.mark.parametrize("strength", [1e-4, 0.1, 3.0, 60.0])
def test_chunks_against_float64(ops, G, H, d, dv, strength):
    gen = torch.Generator(device="cuda").manual_seed(d + dv)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    lens, before = [1, 2, 31, 127, 128, 1, 129, 200, 520], [3, 0, 7, 0, 5, 0, 0, 64, 0]
    T, B = sum(lens), len(lens)
    rows = rnd(T, 2 * G * d + H * dv)
    rows[:, :2 * G * d] *= d ** -0.5
    beta = torch.rand(T, H, device="cuda", generator=gen)
    decay = torch.exp(-strength * torch.rand(T, H, device="cuda", generator=gen))
    if strength > 10:
        decay[::7] = 0.0                                   # an exponential that underflowed
    state = rnd(B + 2, H, dv, d)
    slots = i32([(2 * b + 1) % (B + 2) for b in range(B)])
    cu, ctx = i32([sum(lens[:b]) for b in range(B + 1)]), i32([a + b for a, b in zip(lens, before)])
    tiles = [(b, x) for b, n in enumerate(lens) if n > 1 for x in range(0, n, 128)]
    want, after = torch.zeros(T, H * dv, dtype=torch.float64, device="cuda"), state.double()
    rep, at = H // G, 0
    for b, n in enumerate(lens):
        r = rows[at:at + n].double()
        q, k = (r[:, i * G * d:(i + 1) * G * d].view(n, G, d).repeat_interleave(rep, 1) for i in (0, 1))
        s = int(slots[b])
        o, S = walk(q, k, r[:, 2 * G * d:].view(n, H, dv), decay[at:at + n].double(), beta[at:at + n].double(),
                    state[s].double() if before[b] else torch.zeros_like(after[s]))
        want[at:at + n], after[s] = o.reshape(n, -1), S
        at += n
    got = []
    for chunked in (True, False):
        st, out = state.clone(), torch.full((T, H * dv), float("nan"), device="cuda")
        if chunked:
            scratch = torch.full((ops.linear_scratch_floats(T, B, H, d, dv),), float("nan"), device="cuda")
            assert ops.linear_chunks(rows, beta, decay, st, scratch, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), len(tiles),
                                     cu, ctx, slots, B, G, H, d, dv, out)
            ops.delta_recur(rows, beta, decay, st, cu, ctx, slots, B, G, H, d, dv, out, plain=True, max_len=1)
            assert int(ops.tc_status("cuda")[0]) == 0
        else:
            ops.delta_recur(rows, beta, decay, st, cu, ctx, slots, B, G, H, d, dv, out, plain=True)
        got.append([float((x.double() - y).norm() / y.norm()) for x, y in ((out, want), (st, after))]
                   + [float((x.double() - y).abs().max() / y.abs().max()) for x, y in ((out, want), (st, after))])
    print(f"chunks {['%.1e' % e for e in got[0]]} token by token {['%.1e' % e for e in got[1]]}")
    # products in three tf32 parts are 2^-21 from float32's; up to 96 sums of an accumulator, each cut off at 2^-23
    assert max(got[0][:2]) < 4e-6 and max(got[0][2:]) < 8e-6


def test_refuses_what_it_does_not_take(ops):
    assert not ops.linear_chunks_ok(12, 64) and not ops.linear_chunks_ok(264, 64) and not ops.linear_chunks_ok(64, 260)
    T, H, d, dv = 70, 2, 12, 8
    rows, w, st = torch.randn(T, 2 * H * d + H * dv, device="cuda"), torch.ones(T, H, device="cuda"), torch.zeros(1, H, dv, d, device="cuda")
    out = torch.full((T, H * dv), 7.0, device="cuda")
    scratch = torch.empty(ops.linear_scratch_floats(T, 1, H, d, dv), device="cuda")
    assert not ops.linear_chunks(rows, w, w, st, scratch, i32([0]), i32([0]), 1, i32([0, T]), i32([T]), i32([0]), 1, H, H, d, dv, out)
    assert bool((out == 7.0).all())


@pytest.mark.parametrize("H,d,dv,dtype", [(2, 64, 128, torch.float32), (2, 128, 256, torch.bfloat16), (2, 8, 4, torch.float32), (1, 72, 60, torch.bfloat16), (1, 256, 200, torch.float32)])
def test_retention_against_float64(ops, H, d, dv, dtype):
    """The same with one fixed decay a head, the unit norm and the gate: every store of the epilogue."""
    gen = torch.Generator(device="cuda").manual_seed(d + dv)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    lens, before = [2, 1, 128, 33, 300], [0, 0, 5, 9, 1]
    T, B, eps = sum(lens), len(lens), 1e-6
    rows = rnd(T, H * (2 * d + dv))
    rows[:, :2 * H * d] *= d ** -0.5
    decay = 1.0 - 2.0 ** -(5.0 + torch.arange(H, device="cuda", dtype=torch.float64))
    log2 = decay.log2().float()
    state, gate = rnd(B, H, dv, d), rnd(T, H * dv + 16).to(dtype)[:, 8:-8]
    cu, ctx = i32([sum(lens[:b]) for b in range(B + 1)]), i32([a + b for a, b in zip(lens, before)])
    tiles = [(b, x) for b, n in enumerate(lens) if n > 1 for x in range(0, n, 128)]
    scratch = torch.full((ops.linear_scratch_floats(T, B, H, d, dv),), float("nan"), device="cuda")
    out, st = torch.full((T, H * dv), 7.0, device="cuda", dtype=dtype), state.clone()
    assert ops.linear_retention(rows, log2, st, scratch, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), len(tiles), cu, ctx,
                                i32(list(range(B))), B, gate, eps, H, d, dv, out)
    assert int(ops.tc_status("cuda")[0]) == 0
    at = 0
    for b, n in enumerate(lens):
        if n == 1:                                         # left alone
            assert bool((out[at] == 7.0).all()) and torch.equal(st[b], state[b])
            at += n
            continue
        r = rows[at:at + n].double()
        q, k, v = r[:, :H * d].view(n, H, d), r[:, H * d:2 * H * d].view(n, H, d), r[:, 2 * H * d:].view(n, H, dv)
        ones = torch.ones(n, H, dtype=torch.float64, device="cuda")
        o, S = walk(q, k, v, (2.0 ** log2.double()) * ones, ones, state[b].double() if before[b] else torch.zeros_like(state[b]).double())
        z = gate[at:at + n].double().view(n, H, dv)
        want = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + eps) * z * torch.sigmoid(z)
        got = out[at:at + n].double().view(n, H, dv)
        # the sums as above; a row whose o is small against its terms keeps their error, hence the norm; bfloat16: one rounding
        rel = float((got - want).norm() / want.norm())
        assert rel < (4e-6 if dtype == torch.float32 else 2.5e-3), rel
        assert float((st[b].double() - S).norm() / S.norm()) < 4e-6
        at += n


@pytest.mark.parametrize("lens,chunked", [([255, 1, 3], False), ([256, 1, 3], True), ([1, 1], False)])
def test_mixers_recurrence_takes_chunks_for_long_portions(ops, monkeypatch, lens, chunked):
    """PlainRecurrence: a portion's own length decides; short portions and single tokens of the same step are walked."""
    from types import SimpleNamespace
    from gollmgo_b200.parts import linear_recurrence as L
    from gollmgo_b200.parts.context import Workspace
    G, H, d, dv, T, B = 1, 2, 128, 8, sum(lens), len(lens)
    ws = Workspace(torch.device("cuda"))
    rec = L.PlainRecurrence(SimpleNamespace(workspace=ws, max_tokens=T, max_seqs=B), G, H, d, dv)
    need, = rec.query_tiles()
    rows, beta, decay = (torch.rand(T, w, device="cuda") for w in (2 * G * d + H * dv, H, H))
    state, cu, ctx = torch.rand(B, H, dv, d, device="cuda"), i32([sum(lens[:b]) for b in range(B + 1)]), i32([n + 2 for n in lens])
    tiles = [(b, x) for b, n in enumerate(lens) if n > 1 and n >= need.at_least for x in range(0, n, 128)]
    batch = SimpleNamespace(cu_q_lens=cu, context_lens=ctx, state_slots=i32(list(range(B))), num_seqs=B, q_lens=lens,
                            num_portions=sum(n > 1 for n in lens), num_decode=sum(n == 1 for n in lens),
                            tiles={need: SimpleNamespace(seq=i32([t[0] for t in tiles]), q0=i32([t[1] for t in tiles]), count=len(tiles),
                                                   left_out=sum(1 < n < need.at_least for n in lens))})
    calls, real = [], ops.linear_chunks
    monkeypatch.setattr(ops, "linear_chunks", lambda *a: calls.append(1) or real(*a))
    got, want = [(state.clone(), torch.full((T, H * dv), float("nan"), device="cuda")) for _ in range(2)]
    rec.run(rows, beta, decay, got[0], batch, got[1])
    ops.delta_recur(rows, beta, decay, want[0], cu, ctx, batch.state_slots, B, G, H, d, dv, want[1], plain=True)
    assert bool(calls) == chunked
    for a, b in zip(got, want):                            # (both within the bound above of float64)
        assert float((a - b).norm() / b.norm()) < (8e-6 if chunked else 1e-12)
    walked = [b for b, n in enumerate(lens) if n < need.at_least]
    assert torch.equal(got[0][walked], want[0][walked]) and torch.equal(got[1][lens[0]:], want[1][lens[0]:])


@pytest.mark.parametrize("G,H,d,dv,lens,heads", [(4, 16, 64, 64, [1280, 700, 68], 2), (4, 16, 64, 200, [1280, 700, 68], 2),
                                                 (1, 32, 64, 64, [1280, 700, 68], 4), (1, 32, 64, 128, [2048], 4), (1, 64, 64, 32, [2048, 100], 8)])
def test_several_heads_of_a_block(ops, G, H, d, dv, lens, heads):
    """Steps so long that a block of the rows takes two, four or eight heads of a group: beside the token-by-token kernel."""
    gen = torch.Generator(device="cuda").manual_seed(H + dv)
    T, B = sum(lens), len(lens)
    tiles = [(b, x) for b, n in enumerate(lens) for x in range(0, n, 128)]
    turns = lambda h: -(-len(tiles) * (H // h) // 148) * (4 + 5 * h)  # noqa: E731
    assert min((h for h in (1, 2, 4, 8) if H // G % h == 0), key=turns) == heads
    rows = torch.randn(T, 2 * G * d + H * dv, device="cuda", generator=gen)
    rows[:, :2 * G * d] *= d ** -0.5
    beta, decay = torch.rand(T, H, device="cuda", generator=gen), torch.exp(-0.1 * torch.rand(T, H, device="cuda", generator=gen))
    state = torch.randn(B, H, dv, d, device="cuda", generator=gen)
    cu, ctx, slots = i32([sum(lens[:b]) for b in range(B + 1)]), i32([n + 9 for n in lens]), i32(list(range(B)))
    scratch = torch.full((ops.linear_scratch_floats(T, B, H, d, dv),), float("nan"), device="cuda")
    got, want = [(state.clone(), torch.full((T, H * dv), float("nan"), device="cuda")) for _ in range(2)]
    assert ops.linear_chunks(rows, beta, decay, got[0], scratch, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), len(tiles), cu, ctx,
                             slots, B, G, H, d, dv, got[1])
    ops.delta_recur(rows, beta, decay, want[0], cu, ctx, slots, B, G, H, d, dv, want[1], plain=True)
    assert int(ops.tc_status("cuda")[0]) == 0
    for a, b in zip(got, want):                            # (each within 4e-6 of float64, above)
        assert float((a - b).norm() / b.norm()) < 8e-6


def test_decays_between_tokens_are_rounded_once(ops):
    """Every head writes a single 1 and reads nothing: its state is two to the sum of the logarithms behind that token.  Exponents of -8 to
    -14 in float32, off by half an ulp (4.8e-7) at most: 1.9e-7 in the root mean square after ln 2, exp2f and the weight's 22 bits 1e-7."""
    H, d, dv, T, off = 64, 8, 4, 128, []
    h, one = torch.arange(H, device="cuda"), torch.ones(T, H, device="cuda")
    for seed in range(8):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        decay = torch.exp2(-(0.05 + 0.125 * torch.rand(T, H, device="cuda", generator=gen)))
        at = torch.randint(8, 56, (H,), device="cuda", generator=gen)
        rows = torch.zeros(T, 2 * H * d + H * dv, device="cuda")
        rows[at, H * d + h * d] = 1.0
        rows[at, 2 * H * d + h * dv] = 1.0
        state, out = torch.zeros(1, H, dv, d, device="cuda"), torch.empty(T, H * dv, device="cuda")
        scratch = torch.empty(ops.linear_scratch_floats(T, 1, H, d, dv), device="cuda")
        assert ops.linear_chunks(rows, one, decay, state, scratch, i32([0]), i32([0]), 1, i32([0, T]), i32([T]), i32([0]), 1, H, H, d, dv, out)
        logs = torch.log2(decay).double()
        want = torch.exp2(torch.stack([logs[int(at[i]) + 1:, i].sum() for i in range(H)]))
        off.append(state[0, :, 0, 0].double() / want - 1)
    off = torch.cat(off)
    # measured 2.0e-7 (float64 differences: the same); with a second rounding 3.0e-7
    assert float(off.pow(2).mean().sqrt()) < 2.4e-7 and float(off.abs().max()) < 6.5e-7
