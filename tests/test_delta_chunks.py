"""The gated delta rule in chunks (csrc/delta_chunks.cu) against float64 and beside the token-by-token kernel: chunks of 64 and tiles
of 128 tokens at their edges, carried states, single tokens left alone, decays from none to total, keys that repeat."""
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
        S = S * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - (S * k[t][:, None, :]).sum(-1))
        S = S + u[:, :, None] * k[t][:, None, :]
        out[t] = (S * q[t][:, None, :]).sum(-1)
    return out, S


def make(lens, before, G, H, d, dv, strength, repeat=False):
    gen = torch.Generator(device="cuda").manual_seed(d + dv)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T, B = sum(lens), len(lens)
    rows = rnd(T, 2 * G * d + H * dv)
    qk = rows[:, :2 * G * d].view(T, 2 * G, d)
    if repeat:                                             # every key close to one direction: nothing of the system's matrix is small
        qk[:] = qk * 0.05 + 1.0
    qk /= qk.norm(dim=-1, keepdim=True)
    beta = torch.rand(T, H, device="cuda", generator=gen)
    decay = torch.exp(-strength * torch.rand(T, H, device="cuda", generator=gen))
    if strength > 10:
        decay[::7] = 0.0                                   # an exponential that underflowed
    state = rnd(B + 2, H, dv, d)
    slots = i32([(2 * b + 1) % (B + 2) for b in range(B)])
    cu, ctx = i32([sum(lens[:b]) for b in range(B + 1)]), i32([a + b for a, b in zip(lens, before)])
    tiles = [(b, x) for b, n in enumerate(lens) if n > 1 for x in range(0, n, 128)]
    return rows, beta, decay, state, slots, cu, ctx, tiles


def chunks(ops, rows, beta, decay, st, slots, cu, ctx, tiles, G, H, d, dv):
    T, B = rows.shape[0], len(slots)
    scratch = torch.full((ops.linear_scratch_floats(T, B, H, d, dv),), float("nan"), device="cuda")
    solved = torch.full((ops.delta_solved_floats(T, B, G, H, d),), float("nan"), device="cuda")
    out = torch.full((T, H * dv), float("nan"), device="cuda")
    assert ops.delta_chunks(rows, beta, decay, st, scratch, solved, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), len(tiles),
                            cu, ctx, slots, B, G, H, d, dv, out)
    ops.delta_recur(rows, beta, decay, st, cu, ctx, slots, B, G, H, d, dv, out, max_len=1)
    assert int(ops.tc_status("cuda")[0]) == 0
    return out


@pytest.mark.parametrize("G,H,d,dv", [(1, 4, 128, 128), (2, 4, 64, 128), (3, 3, 96, 16), (2, 2, 32, 64), (1, 2, 128, 256), (2, 2, 64, 144), (1, 8, 32, 32)])
@pytest.mark.parametrize("strength,repeat", [(1e-4, False), (0.1, True), (3.0, False), (60.0, False)])
def test_chunks_against_float64(ops, G, H, d, dv, strength, repeat):
    lens, before = [1, 2, 63, 64, 65, 1, 127, 128, 129, 200, 520], [3, 0, 7, 0, 5, 0, 0, 64, 0, 2, 9]
    rows, beta, decay, state, slots, cu, ctx, tiles = make(lens, before, G, H, d, dv, strength, repeat)
    T, B = sum(lens), len(lens)
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
        st = state.clone()
        if chunked:
            out = chunks(ops, rows, beta, decay, st, slots, cu, ctx, tiles, G, H, d, dv)
        else:
            out = torch.full((T, H * dv), float("nan"), device="cuda")
            ops.delta_recur(rows, beta, decay, st, cu, ctx, slots, B, G, H, d, dv, out)
        got.append([float((x.double() - y).norm() / y.norm()) for x, y in ((out, want), (st, after))]
                   + [float((x.double() - y).abs().max() / y.abs().max()) for x, y in ((out, want), (st, after))])
    print(f"chunks {['%.1e' % e for e in got[0]]} token by token {['%.1e' % e for e in got[1]]}")
    # rows: products in three tf32 parts are 2^-21 from float32's, sums cut off at 2^-23 (test_linear_chunks.py); states: float32
    # sums, of which a token's write goes through at most 64 + d and 64 (2^-24 each, as in the walk)
    assert max(got[0][:2]) < 4e-6 and max(got[0][2:]) < 8e-6


@pytest.mark.parametrize("where", ["q", "k", "v", "beta", "decay"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_bad_values_reach_no_earlier_token(ops, where, bad):
    G, H, d, dv, n, at = 1, 2, 64, 32, 300, 171
    rows, beta, decay, state, slots, cu, ctx, tiles = make([n], [5], G, H, d, dv, 0.1)
    clean = chunks(ops, rows, beta, decay, state.clone(), slots, cu, ctx, tiles, G, H, d, dv)
    if where in "qkv":
        rows[at, {"q": 3, "k": G * d + 3, "v": 2 * G * d + 3}[where]] = bad
    else:
        (beta if where == "beta" else decay)[at, 0] = bad
    out, walked = (torch.full((n, H * dv), 7.0, device="cuda") for _ in range(2))
    st, st2 = state.clone(), state.clone()
    out = chunks(ops, rows, beta, decay, st, slots, cu, ctx, tiles, G, H, d, dv)
    ops.delta_recur(rows, beta, decay, st2, cu, ctx, slots, 1, G, H, d, dv, walked)
    # (a block of eight tokens that has a bad value is solved by substitution: the ones ahead of it agree within the bound above)
    assert bool(torch.isfinite(out[:at]).all()) and float((out[:at] - clean[:at]).norm() / clean[:at].norm()) < 4e-6
    # wherever the walk has no number there is none here, and no fewer rows and columns have one than in the walk, but for those
    # that an infinite value passes by a weight of 0
    fine, wfine = torch.isfinite(out), torch.isfinite(walked)
    assert not bool((fine & ~wfine).any())
    if bad != bad:
        assert torch.equal(fine, wfine)
        assert torch.equal(torch.isfinite(st), torch.isfinite(st2))


def test_refuses_what_it_does_not_take(ops):
    assert not ops.delta_chunks_ok(40, 64) and not ops.delta_chunks_ok(160, 64) and not ops.delta_chunks_ok(64, 24) and not ops.delta_chunks_ok(64, 272)
    T, H, d, dv = 70, 2, 64, 24
    rows, w, st = torch.randn(T, 2 * H * d + H * dv, device="cuda"), torch.ones(T, H, device="cuda"), torch.zeros(1, H, dv, d, device="cuda")
    out = torch.full((T, H * dv), 7.0, device="cuda")
    scratch = torch.empty(ops.linear_scratch_floats(T, 1, H, d, dv), device="cuda")
    solved = torch.empty(ops.delta_solved_floats(T, 1, H, H, d), device="cuda")
    assert not ops.delta_chunks(rows, w, w, st, scratch, solved, i32([0]), i32([0]), 1, i32([0, T]), i32([T]), i32([0]), 1, H, H, d, dv, out)
    assert bool((out == 7.0).all())


def error(x, y):
    return float((x.double() - y).norm() / y.norm())


@pytest.mark.parametrize("G,H,d,dv,lens", [(4, 16, 128, 128, [1280, 768]), (2, 16, 64, 64, [2000, 1500, 700]), (1, 8, 128, 144, [3600]),
                                           (1, 4, 96, 32, [700, 513, 835])])
@pytest.mark.parametrize("fast", [True, False])
def test_no_further_from_float64_than_the_walk(ops, G, H, d, dv, lens, fast):
    """Values and decays as a layer makes them (a step's softplus times 1 to 16, or 1 - 2^-5 to 1 - 2^-13 over the heads), blocks of one, two
    and four heads: float32 sums in another order, not fewer bits."""
    gen = torch.Generator(device="cuda").manual_seed(H + dv)
    rnd, uni = (lambda *s: torch.randn(*s, device="cuda", generator=gen)), (lambda *s: torch.rand(*s, device="cuda", generator=gen))  # noqa: E731
    T, B = sum(lens), len(lens)
    rows = torch.nn.functional.silu(rnd(T, 2 * G * d + H * dv))
    qk = rows[:, :2 * G * d].view(T, 2 * G, d)
    qk /= qk.norm(dim=-1, keepdim=True)
    rows[:, :G * d] *= d ** -0.5
    if fast:
        start = 1e-3 * 100.0 ** uni(H)
        decay = torch.exp(-(1 + 15 * uni(H)) * torch.nn.functional.softplus(rnd(T, H) + start + torch.log(-torch.expm1(-start))))
    else:
        decay = (1.0 - 2.0 ** (-5.0 - 8.0 * torch.arange(H, device="cuda") / (H - 1))).expand(T, H).contiguous()
    beta, state = torch.sigmoid(rnd(T, H)), rnd(B, H, dv, d) * 0.3
    slots, cu, ctx = i32(list(range(B))), i32([sum(lens[:b]) for b in range(B + 1)]), i32([n + 40 for n in lens])
    want, after, at = torch.zeros(T, H * dv, dtype=torch.float64, device="cuda"), state.double(), 0
    for b, n in enumerate(lens):
        r = rows[at:at + n].double()
        q, k = (r[:, i * G * d:(i + 1) * G * d].view(n, G, d).repeat_interleave(H // G, 1) for i in (0, 1))
        o, after[b] = walk(q, k, r[:, 2 * G * d:].view(n, H, dv), decay[at:at + n].double(), beta[at:at + n].double(), after[b])
        want[at:at + n] = o.reshape(n, -1)
        at += n
    st, st2, walked = state.clone(), state.clone(), torch.full((T, H * dv), float("nan"), device="cuda")
    out = chunks(ops, rows, beta, decay, st, slots, cu, ctx, [(b, x) for b, n in enumerate(lens) for x in range(0, n, 128)], G, H, d, dv)
    ops.delta_recur(rows, beta, decay, st2, cu, ctx, slots, B, G, H, d, dv, walked)
    print(f"rows {error(out, want):.2e}, walk {error(walked, want):.2e}; state {error(st, after):.2e}, walk {error(st2, after):.2e}")
    # measured over 40 such steps: rows 0.56 to 1.09 of the walk's error, states 0.42 to 0.76
    assert error(out, want) < 1.25 * error(walked, want) and error(st, after) < error(st2, after)


@pytest.mark.parametrize("where", ["v", "k", "beta"])
def test_bad_values_in_wide_rows(ops, where):
    """The same where a block's rows have 128 and sixteen columns and four heads: what is no number reaches what it reaches in the walk, in
    its chunk and behind it, and the other heads and sequences not at all."""
    G, H, d, dv, lens, at = 2, 8, 128, 144, [700, 2048, 2000], 700 + 1000
    rows, beta, decay, state, slots, cu, ctx, tiles = make(lens, [0, 5, 0], G, H, d, dv, 0.05)
    assert len(tiles) * H >= 222 and H // G % 2 == 0       # (two heads a block)
    clean = chunks(ops, rows, beta, decay, state.clone(), slots, cu, ctx, tiles, G, H, d, dv)
    if where == "beta":
        beta[at, 3] = float("nan")
    else:
        rows[at, {"k": G * d + d + 3, "v": 2 * G * d + 3 * dv + 130}[where]] = float("nan")
    st, st2, walked = state.clone(), state.clone(), torch.full((sum(lens), H * dv), 7.0, device="cuda")
    out = chunks(ops, rows, beta, decay, st, slots, cu, ctx, tiles, G, H, d, dv)
    ops.delta_recur(rows, beta, decay, st2, cu, ctx, slots, len(lens), G, H, d, dv, walked)
    assert torch.equal(torch.isfinite(out), torch.isfinite(walked)) and torch.equal(torch.isfinite(st), torch.isfinite(st2))
    assert bool((~torch.isfinite(out[at:700 + 2048])).any())
    fine = torch.isfinite(out)
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[700 + 2048:], clean[700 + 2048:])
    assert float((out[fine] - clean[fine]).norm() / clean[fine].norm()) < 1e-12
