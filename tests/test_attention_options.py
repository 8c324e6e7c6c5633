"""The tcgen05 prompt attention with the options of the general path (csrc/attention_tc3.cu) against float64: tiles of 128
queries and steps of 128 keys at their edges, portions behind a context, keys and values of every pair of sizes."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
PAGE = 16


@pytest.fixture(scope="module")
def ops():
    from gollmgo_b200.csrc import ops
    return ops


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


OPTIONS = {
    "plain": {}, "capped": {"softcap": 5.0}, "sloped": {"slopes": True, "sink": True, "temperature": (0.1, 64)},
    "window": {"window": 100, "slopes": True}, "chunk": {"chunk": 96, "sink": True}, "both": {"softcap": 8.0, "slopes": True, "window": 150},
}


@pytest.mark.parametrize("option", sorted(OPTIONS))
@pytest.mark.parametrize("d,dv,v_share,out_f32", [(128, 128, 1, False), (64, 128, 2, True), (128, 64, 1, False), (64, 64, 1, True)])
def test_options_against_float64(ops, option, d, dv, v_share, out_f32):
    o = OPTIONS[option]
    gen = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    nkv, group = 2, 4
    nh, nv = nkv * group, nkv // v_share
    lens, starts = [2, 127, 128, 129, 300], [0, 130, 0, 250, 37]
    ctx = [a + b for a, b in zip(starts, lens)]
    T, B, scale = sum(lens), len(lens), d ** -0.5
    q = rnd(T, nh * d + 8).to(torch.bfloat16)
    per = [-(-c // PAGE) for c in ctx]
    pages = torch.randperm(sum(per) + 3, device="cuda", generator=gen).to(torch.int32)
    table = torch.full((B, max(per)), -1, dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(per):
        table[b, :n] = pages[at:at + n]
        at += n
    # rows past a context, and pages nobody holds, are NaN: no result may depend on them
    kc = torch.full((sum(per) + 3, nkv, PAGE, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    vc = torch.full((sum(per) + 3, nv, PAGE, dv), float("nan"), dtype=torch.bfloat16, device="cuda")
    keys, values = [], []
    for b, n in enumerate(ctx):
        k, v = rnd(n, nkv, d).to(torch.bfloat16), rnd(n, nv, dv).to(torch.bfloat16)
        keys.append(k.double())
        values.append(v.double())
        for j in range(n):
            kc[table[b, j // PAGE], :, j % PAGE] = k[j]
            vc[table[b, j // PAGE], :, j % PAGE] = v[j]
    slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / nh) for h in range(nh)], device="cuda") if o.get("slopes") else None
    sink = rnd(nh) if o.get("sink") else None
    tiles = [(b, x) for b, n in enumerate(lens) for x in range(0, n, 128)]
    cu = i32([sum(lens[:i]) for i in range(B + 1)])
    out = torch.empty(T, nh * dv, dtype=torch.float32 if out_f32 else torch.bfloat16, device="cuda")
    t0, t1 = i32([t[0] for t in tiles]), i32([t[1] for t in tiles])
    ops.attn_prefill_x(q, q.stride(0), kc, vc, table, table.shape[1], cu, i32(ctx), t0, t1, 0, out, nh, nkv, d, dv, v_share, PAGE,
                       o.get("window", 0), scale, o.get("softcap", 0.0), chunk=o.get("chunk", 0), sink=sink, slopes=slopes,
                       temperature=o.get("temperature"), tile128_seq=t0, tile128_q0=t1, num_tiles128=len(tiles))
    torch.cuda.synchronize()
    assert int(ops.tc_status("cuda")[0]) == 0
    at = 0
    for b, n in enumerate(lens):
        qb = q[at:at + n, :nh * d].double().view(n, nh, d)
        i = torch.arange(starts[b], ctx[b], device="cuda")[:, None]
        j = torch.arange(ctx[b], device="cuda")[None, :]
        seen = j <= i
        if o.get("window"):
            seen = seen & (i - j < o["window"])
        if o.get("chunk"):
            seen = seen & (j >= i // o["chunk"] * o["chunk"])
        for h in range(nh):
            s = (qb[:, h] @ keys[b][:, h // group].T) * scale
            if o.get("temperature"):
                c, every = o["temperature"]
                s = s * (1 + c * torch.log(torch.floor((i + 1.0) / every) + 1))
            if o.get("softcap"):
                s = o["softcap"] * torch.tanh(s / o["softcap"])
            if slopes is not None:
                s = s - slopes[h].double() * (i - j)
            s = s.masked_fill(~seen, -math.inf)
            top = s.max(-1, keepdim=True).values
            e = torch.exp(s - top)
            z = e.sum(-1, keepdim=True) + (torch.exp(sink[h].double() - top) if sink is not None else 0.0)
            want = (e / z) @ values[b][:, h // group // v_share]
            got = out[at:at + n, h * dv:(h + 1) * dv].double()
            # weights and results rounded to bfloat16 (2^-9 each), a cap's tanh to 2^-11 of the cap in the exponent
            assert float((got - want).abs().max() / want.abs().max()) < 1.5e-2, (b, h)
        at += n
