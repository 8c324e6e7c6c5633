"""The convolution, gate and norm kernels of the recurrent layers and the cache write of the general attention path, eight or
four values a thread, against float64: sequences that begin and end inside a block of tokens, carried windows, single tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from gollmgo_b200.csrc import ops
    return ops


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def conv(x, w, carried, bias=None):
    """silu of the causal convolution over the rows x, and the last inputs."""
    full = torch.cat([carried, x])
    n = w.shape[1]
    y = sum(full[j:j + x.shape[0]] * w[:, j] for j in range(n))
    y = y if bias is None else y + bias
    return y * torch.sigmoid(y), full[full.shape[0] - (n - 1):]


def near(got, want, tol):
    """Within tol of the largest value (float32 sums of a few values; the activation type where that is bfloat16)."""
    err = float((got.double() - want).abs().max() / want.abs().max())
    assert err <= tol, f"{err:.2e}"


# (tokens of each sequence, tokens it had before): around the tokens of a block; a step of single tokens; as many tokens as
# sequences, though some have two and some none
STEPS = [([1, 7, 8, 9, 2, 17, 30], [0, 5, 0, 2, 1, 0, 3]), ([1] * 11, [0, 1, 2, 3, 9, 0, 5, 40, 1, 0, 2]), ([64], [0]), ([1, 33], [4, 0]),
         ([2, 0, 1], [3, 4, 0]),
         # as many tokens as blocks of four, eight and sixteen take (two blocks a multiprocessor of one group of channels)
         ([1290, 3, 17], [0, 2, 0]), ([2480, 9], [5, 0]), ([4750, 33, 16], [1, 0, 7])]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("step", range(len(STEPS)))
def test_delta_and_ssm_prep(ops, dtype, taps, step):
    lens, before = STEPS[step]
    gen = torch.Generator(device="cuda").manual_seed(17 * taps + step)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T, B = sum(lens), len(lens)
    cu, ctx = i32([sum(lens[:i]) for i in range(B + 1)]), i32([a + b for a, b in zip(lens, before)])
    slots = i32([(3 * i + 1) % (B + 1) if (B + 1) % 3 else i for i in range(B)])

    def rows_of(x, w, state, bias=None):
        ys, at = [], 0
        after = state.double().clone()
        for b, n in enumerate(lens):
            s = int(slots[b])
            carried = state[s].double() if before[b] else torch.zeros_like(state[s]).double()
            y, last = conv(x[at:at + n].double(), w.double(), carried, bias)
            ys.append(y)
            after[s] = last
            at += n
        return torch.cat(ys), after

    for G, H, d, dv in [(2, 4, 64, 24), (1, 3, 128, 40), (2, 2, 256, 128), (3, 3, 32, 4)]:
        C = 2 * G * d + H * dv
        x, w = rnd(T, C + 8).to(dtype), rnd(C, taps)
        state = rnd(B + 1, taps - 1, C)
        zb, za, a_log, dt_b = rnd(T, H), rnd(T, H), rnd(H), rnd(H)
        y, after = rows_of(x[:, :C], w, state)
        q, k, v = y[:, :G * d].view(T, G, d), y[:, G * d:2 * G * d].view(T, G, d), y[:, 2 * G * d:]
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        out, beta, decay = (torch.empty(T, n, device="cuda") for n in (C, H, H))
        ops.delta_prep(x, w, state, zb, za, a_log, dt_b, cu, ctx, slots, B, G, H, d, dv, out, beta, decay)
        for got, want in ((out[:, :G * d], q.reshape(T, -1)), (out[:, G * d:2 * G * d], k.reshape(T, -1)), (out[:, 2 * G * d:], v)):
            near(got, want, 5e-6)
        near(beta, torch.sigmoid(zb.double()), 1e-6)
        near(decay, torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus((za + dt_b).double())), 5e-6)
        near(state, after, 1e-7)

    for H, P, G, N in [(4, 16, 1, 64), (4, 8, 2, 24)]:
        inner, Cc = H * P, H * P + 2 * G * N
        width = -(-(inner + Cc + H) // 8) * 8
        proj, w, bias = rnd(T, width).to(dtype), rnd(Cc, taps), rnd(Cc)
        state, a_log, dt_b = rnd(B + 1, taps - 1, Cc), rnd(H), rnd(H)
        y, after = rows_of(proj[:, inner:inner + Cc], w, state, bias.double())
        cbx, dt, decay = (torch.empty(T, n, device="cuda") for n in (Cc, H, H))
        ops.ssm_prep(proj, w, bias, state, a_log, dt_b, cu, ctx, slots, B, H, P, G, N, cbx, dt, decay)
        near(cbx, torch.cat([y[:, inner + G * N:], y[:, inner:inner + G * N], y[:, :inner]], 1), 5e-6)
        step_size = torch.nn.functional.softplus(proj[:, inner + Cc:inner + Cc + H].double() + dt_b.double())
        near(dt, step_size, 5e-6)
        near(decay, torch.exp(-torch.exp(a_log.double()) * step_size), 5e-6)
        near(state, after, 1e-7)


@pytest.mark.parametrize("lens", [[5, 20], [1, 1, 1]])
def test_rows_behind_the_last_sequence_change_nothing(ops, lens):
    """More rows than the sequences have tokens: the sequences' rows and windows are as without them."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    G, H, d, dv, T, B, more = 1, 3, 32, 4, sum(lens), len(lens), 19
    C = 2 * G * d + H * dv
    x, w = torch.randn(T + more, C, device="cuda", generator=gen), torch.randn(C, 4, device="cuda", generator=gen)
    zb, za, a_log, dt_b = (torch.randn(*s, device="cuda", generator=gen) for s in ((T + more, H), (T + more, H), (H,), (H,)))
    cu, ctx, slots = i32([sum(lens[:b]) for b in range(B + 1)]), i32([n + 3 for n in lens]), i32(list(range(B)))
    start = torch.randn(B, 3, C, device="cuda", generator=gen)
    got = []
    for rows in (T, T + more):
        state, out, beta, decay = start.clone(), *(torch.empty(rows, n, device="cuda") for n in (C, H, H))
        ops.delta_prep(x[:rows], w, state, zb[:rows], za[:rows], a_log, dt_b, cu, ctx, slots, B, G, H, d, dv, out, beta, decay)
        got.append((out[:T], beta[:T], decay[:T], state))
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T", [1, 3, 300])
def test_gated_norms(ops, dtype, T):
    gen = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    tol = 5e-6 if dtype == torch.float32 else 4e-3           # a bfloat16 result is rounded once: half of 2^-7
    for H, dv, act in [(3, 4, "silu"), (5, 128, "silu"), (2, 132, "sigmoid"), (3, 512, "silu"), (2, 30, "silu"), (1, 520, "silu")]:
        o, gate, w = rnd(T, H * dv), rnd(T, H * dv + 8).to(dtype), rnd(dv)
        out = torch.empty(T, H * dv, dtype=dtype, device="cuda")
        z = gate[:, :H * dv].double().view(T, H, dv)
        unit = o.double().view(T, H, dv)
        unit = unit * torch.rsqrt((unit * unit).mean(-1, keepdim=True) + 1e-6)
        g = torch.sigmoid(z) * (z if act == "silu" else 1.0)
        for weight in (w, None):
            ops.delta_out(o, gate[:, :H * dv], weight, 1e-6, H, dv, out, act)
            near(out, (unit * g * (1.0 if weight is None else w.double())).reshape(T, -1), tol)
    for H, P, parts in [(4, 16, 1), (8, 64, 4), (64, 64, 1), (3, 10, 3), (96, 64, 2)]:
        inner = H * P
        y, cbx, z = rnd(T, inner), rnd(T, inner + 16), rnd(T, inner).to(dtype)
        D, w = rnd(H), rnd(inner)
        out = torch.empty(T, inner, dtype=dtype, device="cuda")
        ops.ssm_out(y, cbx, 16, z, D, w, 1e-6, H, P, parts, out)
        zd = z.double()
        v = (y.double() + D.double().repeat_interleave(P) * cbx[:, 16:].double()) * zd * torch.sigmoid(zd)
        v = v.view(T, parts, -1)
        near(out, (v * torch.rsqrt((v * v).mean(-1, keepdim=True) + 1e-6)).view(T, -1) * w.double(), tol)


@pytest.mark.parametrize("with_bias", [False, True])
@pytest.mark.parametrize("nh,nkv,d,nv,dv,rot", [(4, 2, 128, 2, 64, 64), (3, 1, 64, 1, 128, 0), (2, 2, 32, 0, 32, 32), (4, 2, 40, 2, 24, 16)])
def test_rotation_and_cache_write(ops, nh, nkv, d, nv, dv, rot, with_bias):
    """The eight-value kernel and the general one (reached with a row stride that is not a multiple of eight) agree."""
    gen = torch.Generator(device="cuda").manual_seed(d)
    T, page, W = 21, 16, (nh + nkv) * d + nv * dv
    table = 10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64, device="cuda") * 2 / rot) if rot else None
    pos, slots = i32([5 * t + 3 for t in range(T)]), i32([(7 * t) % 32 if t % 6 else -1 for t in range(T)])
    bias = torch.randn(W, device="cuda", generator=gen) if with_bias else None
    rows = torch.randn(T, W, device="cuda", generator=gen).to(torch.bfloat16)
    got = []
    for stride in (W + 8, W + 1):
        qkv = torch.zeros(T, stride, dtype=torch.bfloat16, device="cuda")
        qkv[:, :W] = rows
        kc = torch.zeros(2, nkv, page, d, dtype=torch.bfloat16, device="cuda")
        vc = torch.zeros(2, max(nv, 1), page, dv, dtype=torch.bfloat16, device="cuda")
        ops.rope_kv_write_x(qkv, pos, slots, table, 1.25, bias, kc, vc, nh, nkv, d, nv, dv, page, False, True)
        got.append((qkv[:, :W], kc, vc))
    for a, b in zip(*got):
        # the same products, contracted differently by the compiler: a bfloat16 step at most
        torch.testing.assert_close(a.float(), b.float(), rtol=2 ** -7, atol=1e-6)
