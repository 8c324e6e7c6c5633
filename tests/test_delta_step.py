"""A step of one token a sequence of the gated delta rule in one kernel (delta_step in csrc/delta_rule.cu) beside the three it replaces:
every size it takes, heads alone and shared, fresh, carried and padded sequences, two to four taps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from gollmgo_b200.csrc import ops
    return ops


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("G,H,d,dv", [(2, 2, 64, 64), (1, 2, 128, 64), (2, 8, 128, 128), (1, 8, 64, 128), (3, 6, 64, 256), (2, 4, 128, 256)])
@pytest.mark.parametrize("taps,act", [(4, "silu"), (3, "sigmoid"), (2, "silu")])
def test_step_against_three_kernels(ops, G, H, d, dv, taps, act):
    gen = torch.Generator(device="cuda").manual_seed(d + dv + taps)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    B, C = 5, 2 * G * d + H * dv
    proj = rnd(B, C + H * dv + 8).bfloat16()
    x, gate = proj, proj[:, C + 8:]
    conv_w, norm_w = rnd(C, taps), rnd(dv)
    ba, a_log, dt_bias = rnd(B, 2 * H), rnd(H), rnd(H)
    slots, ctx, cu = i32([3, 0, -1, 5, 1]), i32([4, 1, 9, 2, 700]), i32(list(range(B + 1)))      # a fresh one, a padded one
    state, window = rnd(6, H, dv, d), rnd(6, taps - 1, C)
    got = []
    for one in (True, False):
        st, win, y = state.clone(), window.clone(), torch.zeros(B, H * dv, device="cuda", dtype=torch.bfloat16)
        if one:
            assert ops.delta_step(x, conv_w, win, ba[:, :H], ba[:, H:], a_log, dt_bias, st, cu, ctx, slots, B, G, H, d, dv, gate, norm_w, 1e-6, y, act)
        else:
            qkv, beta, decay, o = (torch.zeros(B, w, device="cuda") for w in (C, H, H, H * dv))
            ops.delta_prep(x, conv_w, win, ba[:, :H], ba[:, H:], a_log, dt_bias, cu, ctx, slots, B, G, H, d, dv, qkv, beta, decay)
            ops.delta_recur(qkv, beta, decay, st, cu, ctx, slots, B, G, H, d, dv, o)
            ops.delta_out(o, gate, norm_w, 1e-6, H, dv, y, act)
        got.append((st, win, y.float()))
    assert torch.equal(got[0][1], got[1][1])               # the window holds inputs
    untouched = [s for s in range(6) if s not in (3, 0, 5, 1)]
    assert torch.equal(got[0][0][untouched], state[untouched])
    # float32 sums of up to 128 values in another order; rows: one rounding to bfloat16 that may fall on the other side
    assert float((got[0][0] - got[1][0]).norm() / got[1][0].norm()) < 1e-6
    real = [0, 1, 3, 4]
    assert float((got[0][2][real] - got[1][2][real]).norm() / got[1][2][real].norm()) < 1e-3
    assert bool(torch.isfinite(got[0][2]).all())


def test_refuses_what_it_does_not_take(ops):
    G, H, d, dv, B, taps = 1, 3, 64, 64, 2, 4              # three heads share one of q and k
    C = 2 * G * d + H * dv
    z = lambda *s: torch.zeros(*s, device="cuda")  # noqa: E731
    x, y = z(B, C + H * dv).bfloat16(), torch.full((B, H * dv), 7.0, device="cuda", dtype=torch.bfloat16)
    assert not ops.delta_step(x, z(C, taps), z(B, taps - 1, C), z(B, H), z(B, H), z(H), z(H), z(B, H, dv, d), i32([0, 1, 2]), i32([1, 1]), i32([0, 1]),
                              B, G, H, d, dv, x[:, C:], z(dv), 1e-6, y)
    assert bool((y == 7.0).all())


@pytest.mark.parametrize("M,split,more,K", [(1, 16, 1, 64), (4, 5120, 32, 2048), (16, 40, 16, 200), (9, 200, 33, 520)])
@pytest.mark.parametrize("normed", [False, True])
def test_two_products_in_one_launch(ops, M, split, more, K, normed):
    """gemm_small_m with a float32 tail beside the two products, also behind a norm folded into x."""
    gen = torch.Generator(device="cuda").manual_seed(split)
    x = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
    w = torch.randn(split + more, K, device="cuda", generator=gen).bfloat16() * K ** -0.5
    kw = {}
    if normed:
        parts = torch.rand(-(-K // 16), 16, device="cuda", generator=gen) + 1.0
        kw = dict(in_partials=parts, hidden=K, eps=1e-6)
    out, tail = torch.empty(M, split, device="cuda", dtype=torch.bfloat16), torch.empty(M, more, device="cuda")
    ops.gemm_small_m_tail(x, w, out, tail, **kw)
    a, b = torch.empty_like(out), torch.empty_like(tail)
    ops.gemm_small_m(x, w[:split].contiguous(), a, **kw)
    ops.gemm_small_m(x, w[split:].contiguous(), b, **kw)
    # the same float32 sums; a row's block may start elsewhere along K
    assert float((tail - b).norm() / b.norm()) < 1e-6
    assert float((out.float() - a.float()).norm() / a.float().norm()) < 1e-3


@pytest.mark.parametrize("M", [1, 16, 17])
@pytest.mark.parametrize("N", [64, 4736])
def test_layer_product_with_a_tail(ops, M, N):
    """linear_with_tail: one launch up to sixteen tokens, two products beyond and where the weights are not stored together."""
    from gollmgo_b200.parts.linear import linear_with_tail
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, 256, device="cuda", generator=gen).bfloat16()
    w = torch.randn(N + 32, 256, device="cuda", generator=gen).bfloat16() / 16
    got = []
    for together in (w, None):
        out, tail = torch.empty(M, N, device="cuda", dtype=torch.bfloat16), torch.empty(M, 32, device="cuda")
        a, b = linear_with_tail(x, together, w[:N], w[N:], out, tail)
        assert a is out and b is tail
        got.append((out.float(), tail))
    # the same float32 sums in another order, and roundings to bfloat16 that fall on the other side
    assert float((got[0][1] - got[1][1]).norm() / got[1][1].norm()) < 1e-6
    assert float((got[0][0] - got[1][0]).norm() / got[1][0].norm()) < 1e-3


def test_steps_that_keep_three_kernels():
    """The sizes at which one kernel was measured to be the slower form (the rule's edges)."""
    from gollmgo_b200.parts.gated_delta import one_kernel
    assert one_kernel(1, 4, 4, 64, 64) and one_kernel(32, 4, 16, 128, 128) and one_kernel(64, 16, 16, 64, 64)
    assert one_kernel(8, 6, 48, 64, 64) and not one_kernel(16, 6, 48, 64, 64) and not one_kernel(64, 8, 32, 64, 64)
    assert one_kernel(16, 1, 8, 128, 128) and not one_kernel(32, 1, 8, 128, 128)
    assert one_kernel(16, 4, 16, 64, 256) and not one_kernel(32, 4, 16, 64, 256) and not one_kernel(16, 1, 8, 64, 256)
    assert one_kernel(8, 1, 8, 128, 256) and not one_kernel(4, 1, 8, 128, 256) and not one_kernel(1, 2, 2, 128, 256)
