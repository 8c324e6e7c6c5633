"""Infinities and NaN in the chunk form of the linear recurrence (csrc/linear_chunks.cu): they reach the rows and states that they
reach token by token, no earlier token and no other sequence."""
import pytest
import torch

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("G,H,d,dv", [(1, 4, 128, 64), (2, 2, 64, 128), (2, 2, 128, 132)])
@pytest.mark.parametrize("where", ["v", "k", "q", "beta", "decay"])
@pytest.mark.parametrize("bad", [INF, -INF, NAN])
def test_bad_values_reach_what_they_reach_token_by_token(G, H, d, dv, where, bad):
    from gollmgo_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(d + dv)
    lens = [300, 140]
    T, B = sum(lens), len(lens)
    rows = torch.randn(T, 2 * G * d + H * dv, device="cuda", generator=gen)
    rows[:, :2 * G * d] *= d ** -0.5
    beta, decay = torch.rand(T, H, device="cuda", generator=gen), torch.exp(-0.02 * torch.rand(T, H, device="cuda", generator=gen))
    for t in (37, 166, 167):                               # of the first sequence: inside a chunk's first, second and third 32 tokens
        if where in "qkv":
            rows[t, {"q": 5, "k": G * d + 5, "v": 2 * G * d + (H - 1) * dv + 9}[where]] = bad
        elif where == "beta" or bad != bad:
            (beta if where == "beta" else decay)[t, H - 1] = bad
        else:
            decay[t, H - 1] = abs(bad)                     # (a decay is no negative number)
    state = torch.randn(B, H, dv, d, device="cuda", generator=gen)
    cu, ctx, slots = i32([0, 300, 440]), i32([300 + 9, 140]), i32([1, 0])
    tiles = [(b, x) for b, n in enumerate(lens) for x in range(0, n, 128)]
    got, want = [(state.clone(), torch.full((T, H * dv), 7.0, device="cuda")) for _ in range(2)]
    scratch = torch.full((ops.linear_scratch_floats(T, B, H, d, dv),), NAN, device="cuda")
    assert ops.linear_chunks(rows, beta, decay, got[0], scratch, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), len(tiles), cu, ctx,
                             slots, B, G, H, d, dv, got[1])
    ops.delta_recur(rows, beta, decay, want[0], cu, ctx, slots, B, G, H, d, dv, want[1], plain=True)
    assert int(ops.tc_status("cuda")[0]) == 0
    for a, b in zip(got, want):
        fine = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), fine)
        assert bool(fine.any())
        # (both within 8e-6 of float64 in the largest value: tests/test_linear_chunks.py)
        assert float((a[fine] - b[fine]).abs().max()) <= 1.6e-5 * float(b[fine].abs().max())


@pytest.mark.parametrize("dv,dtype", [(64, torch.float32), (200, torch.bfloat16)])
def test_retention_rows_before_a_bad_value_stay(dv, dtype):
    from gollmgo_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(dv)
    H, d, T, bad = 2, 64, 200, 45
    rows = torch.randn(T, H * (2 * d + dv), device="cuda", generator=gen)
    gate = torch.randn(T, H * dv, device="cuda", generator=gen).to(dtype)
    log2 = torch.tensor([0.97, 0.999], device="cuda").log2()
    outs = []
    for value in (None, NAN, INF):
        x = rows.clone()
        if value is not None:
            x[bad, 2 * H * d + dv + 3] = value             # head 1
        st, out = torch.zeros(1, H, dv, d, device="cuda"), torch.empty(T, H * dv, device="cuda", dtype=dtype)
        scratch = torch.full((ops.linear_scratch_floats(T, 1, H, d, dv),), NAN, device="cuda")
        assert ops.linear_retention(x, log2, st, scratch, i32([0, 0]), i32([0, 128]), 2, i32([0, T]), i32([T]), i32([0]), 1, gate, 1e-6, H, d,
                                    dv, out)
        outs.append(out.view(T, H, dv))
    for got in outs[1:]:
        assert torch.equal(got[:, 0], outs[0][:, 0]) and torch.equal(got[:bad, 1], outs[0][:bad, 1])
        assert not bool(torch.isfinite(got[bad:, 1]).any())            # (a row's norm takes in all its columns)
