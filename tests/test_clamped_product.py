"""The grouped product with the clamped gated activation in its epilogue (csrc/gemm_tc.cu) against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,inter,limit,alpha,shift", [(8, 8, 0.5, 1.702, 1.0), (64, 128, 7.0, 1.702, 1.0), (200, 136, 1.0, 1.0, 0.0), (72, 264, 2.0, 0.5, -1.0)])
def test_clamped_activation_in_the_product(K, inter, limit, alpha, shift):
    from gollmgo_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(K + inter)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()  # noqa: E731
    groups, tiles = 3, [2, -1, 0, 2, 1]
    x, w = rnd(128 * len(tiles), K), rnd(groups, 2 * inter, K) * K ** -0.5 * 2
    out = torch.full((x.shape[0], inter), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tc_grouped(x, w, out, torch.tensor(tiles, dtype=torch.int32, device="cuda"), groups, gated=True, clamped=(limit, alpha, shift))
    assert int(ops.tc_status("cuda")[0]) == 0
    for i, g in enumerate(tiles):
        got = out[128 * i:128 * i + 128]
        if g < 0:
            assert bool((got == 7.0).all())                # a block of no group is left alone
            continue
        z = x[128 * i:128 * i + 128].double() @ w[g].double().T
        gate, up = z[:, :inter].clamp(max=limit), z[:, inter:].clamp(-limit, limit)
        want = gate * torch.sigmoid(alpha * gate) * (up + shift)
        # one rounding to bfloat16 (2^-9 of the value), and float32 sums over K whose terms add up to a few units
        assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())


def test_clamped_activation_refuses_factors_on_rows():
    from gollmgo_b200.csrc import ops
    x, w, out = (torch.zeros(*s, device="cuda", dtype=torch.bfloat16) for s in ((128, 8), (1, 16, 8), (128, 8)))
    rows, tiles = torch.zeros(128, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    with pytest.raises(ops.KernelError):
        ops.gemm_tc_grouped(x, w, out, tiles, 1, gated=True, row_entry=rows, row_scale=torch.ones(128, device="cuda"), clamped=(1.0, 1.0, 0.0))
    with pytest.raises(ops.KernelError):
        ops.gemm_tc_grouped(x, w[:, :8], out, tiles, 1, clamped=(1.0, 1.0, 0.0))
