"""The work that is timed when this engine's speed is compared: single layers of the registered designs through the parts
registry (``build_mixer`` / ``build_feed_forward``, ``CacheManager``, ``BatchBuilder``), token selection through ``Sampler``, and
whole steps through ``ModelRunner.step``; bfloat16, the serving mode.  Layer sizes are those of ``gollmgo_b200/bench_shapes``.

A prompt case calls the layer as a prompt step does.  A step of single decoded tokens is captured in a CUDA graph once and
replayed, as the engine does with such steps.  Weights, inputs and cached state come from the seed alone.

``exact`` restates every layer in float64 with plain torch operations.
"""
import hashlib
import math

import torch

EPS = 1e-6
PAGE = 16
BF16, F64 = torch.bfloat16, torch.float64


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a whole serving step of a Llama decoder: eight requests at a 2048-token context each get their next token
        dict(name="model_decode", path="model", hidden=4096, layers=4, heads=32, kv=8, dim=128, ff=14336, vocab=32768,
             seqs=8, context=2048, new=1),
        # the same model reads one prompt in one step
        dict(name="model_prompt", path="model", hidden=4096, layers=4, heads=32, kv=8, dim=128, ff=14336, vocab=32768,
             seqs=1, context=0, new=2048),
        # a busy server: the attention layer of 64 decoding requests with contexts of 1700 to 4096 tokens
        dict(name="attention_decode", path="attention", hidden=4096, heads=32, kv=8, dim=128, window=0, softcap=0.0, sloped=False,
             rot=128, seqs=64, context=4096, new=1),
        # a prompt in a layer with a sliding window, a bias by distance, a sink and a query temperature (Rimidra's)
        dict(name="attention_prompt", path="attention", hidden=4096, heads=32, kv=8, dim=128, window=1024, softcap=0.0, sloped=True,
             rot=0, seqs=1, context=0, new=2048),
        # two prompts of different length in a gated delta rule (Bevuvik's right branch)
        dict(name="delta_prompt", path="delta", hidden=2048, heads=16, kv=4, dim=128, vdim=128, conv=4, seqs=2, new=2048),
        # the smallest call: a few decoding requests in one recurrent layer
        dict(name="delta_decode", path="delta", hidden=2048, heads=16, kv=4, dim=128, vdim=128, conv=4, seqs=4, new=4),
        # a prompt in a state-space layer (Fapudra's)
        dict(name="ssm_prompt", path="ssm", hidden=2048, heads=64, vdim=64, state=128, groups=1, conv=4, seqs=1, new=2048),
        # a prompt in a selective scan (Matusun's)
        dict(name="scan_prompt", path="scan", hidden=2048, inner=4096, state=16, rank=128, conv=4, seqs=1, new=2048),
        # prompts of an odd total length in a retention layer (Rimidra's)
        dict(name="retention_prompt", path="retention", hidden=2048, heads=16, dim=128, vdim=256, seqs=3, new=2011),
        # a prompt's tokens in a mixture of experts (Fapudra's: clamped activation, choice inside groups)
        dict(name="moe_prompt", path="moe", kind="clamped", hidden=2048, ff=4096, experts=8, top=2, tokens=2048),
        # the decoded tokens of sixteen requests in a mixture of experts (Rimidra's: weighted inputs, gated shared expert)
        dict(name="moe_decode", path="moe", kind="weigh_input", hidden=2048, ff=4096, experts=8, top=2, tokens=16),
        # the next tokens of 64 requests from a vocabulary of 128 k, each with its own temperature, top-k and top-p
        dict(name="sample", path="sample", rows=64, vocab=128256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["model", "attention", "attention", "delta", "delta", "ssm", "scan", "retention", "moe", "moe", "sample"])
    wide = rng.random() < 0.4
    hidden = 4096 if wide else 2048
    if path == "model":
        decode = rng.random() < 0.5
        c = dict(path=path, hidden=hidden, layers=rng.randint(1, 4), heads=hidden // 128, kv=rng.choice([1, 4, 8]), dim=128,
                 ff=14336 if wide else 8192, vocab=32768)
        if decode:
            return dict(c, seqs=_log(rng, 1, 8), context=_log(rng, 64, 2048), new=1)
        return dict(c, seqs=rng.randint(1, 4), context=0, new=_log(rng, 24, 2048))
    if path == "attention":
        c = dict(path=path, hidden=hidden, heads=hidden // 128, kv=rng.choice([4, 8]), dim=128)
        kind = rng.choice(["plain", "plain", "capped", "sloped", "sloped"])
        c.update(window=1024 if kind == "sloped" else 0, softcap=30.0 if kind == "capped" else 0.0, sloped=kind == "sloped",
                 rot={"plain": 128, "capped": 64, "sloped": 0}[kind])
        if rng.random() < 0.4:
            return dict(c, seqs=_log(rng, 1, 64), context=_log(rng, 128, 4000), new=1)
        return dict(c, seqs=rng.randint(1, 4), context=0, new=_log(rng, 40, 2048))
    if path in ("delta", "ssm", "scan", "retention"):
        if rng.random() < 0.25:
            seqs = _log(rng, 1, 64)
            new = seqs                                     # a token each
        else:
            seqs = rng.randint(1, 6)
            new = _log(rng, 20, 2048)
        if path == "delta":
            return dict(path=path, hidden=hidden, heads=hidden // 128, kv=rng.choice([4, 8]), dim=rng.choice([64, 128, 128]), vdim=128,
                        conv=4, seqs=seqs, new=new)
        if path == "ssm":
            return dict(path=path, hidden=2048, heads=64, vdim=64, state=rng.choice([64, 128]), groups=rng.choice([1, 4, 8]), conv=4,
                        seqs=seqs, new=new)
        if path == "scan":
            return dict(path=path, hidden=2048, inner=4096, state=16, rank=rng.choice([64, 128]), conv=4, seqs=seqs, new=new)
        return dict(path=path, hidden=2048, heads=16, dim=128, vdim=rng.choice([128, 256]), seqs=seqs, new=new)
    if path == "moe":
        kind = rng.choice(["clamped", "weigh_input", "relu2"])
        return dict(path=path, kind=kind, hidden=2048, ff=6144 if kind == "relu2" else rng.choice([1024, 4096]), experts=rng.choice([8, 16]),
                    top=2, tokens=_log(rng, 1, 1800))
    return dict(path=path, rows=_log(rng, 1, 64), vocab=rng.choice([32000, 32768, 128256]))


# ---------------------------------------------------------------- inputs
def _lens(total, n):
    """``total`` tokens over n sequences of different length, at least one each."""
    n = min(n, total)
    w = [3 + (5 * j + 2) % 7 for j in range(n)]
    lens = [max(1, total * x // sum(w)) for x in w]
    i = 0
    while sum(lens) != total:
        step = 1 if sum(lens) < total else -1
        if lens[i % n] + step >= 1:
            lens[i % n] += step
        i += 1
    return lens


def _contexts(c):
    """Tokens that each decoding request already holds."""
    return [max(1, c["context"] - (c["context"] * ((3 * j) % 8)) // 12) for j in range(c["seqs"])]


class _Draws:
    def __init__(self, seed, salt):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}/{salt}".encode()).digest()[:7], "little"))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=BF16):
        return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=self.gen).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=BF16):
        return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=self.gen).to(dtype)

    def matrix(self, rows, cols):
        return self.normal(rows, cols, std=cols ** -0.5)

    def taps(self, channels, n):
        return self.normal(channels, n, std=n ** -0.5)

    def steps(self, *shape):
        """Biases whose softplus lies between 1/1000 and 1/10, evenly over the logarithm, as state-space layers start with."""
        dt = torch.exp(self.uniform(*shape, lo=math.log(1e-3), hi=math.log(0.1), dtype=torch.float32))
        return (dt + torch.log(-torch.expm1(-dt))).to(BF16)


def _weights(c, seed):
    d = _Draws(seed, "weights")
    H = c.get("hidden")
    if c["path"] == "attention":
        w = {"q_proj.weight": d.matrix(c["heads"] * c["dim"], H), "k_proj.weight": d.matrix(c["kv"] * c["dim"], H),
             "v_proj.weight": d.matrix(c["kv"] * c["dim"], H), "o_proj.weight": d.matrix(H, c["heads"] * c["dim"])}
        if c["sloped"]:
            w["sink"] = d.normal(c["heads"])
        return w
    if c["path"] == "delta":
        qk, vv = c["kv"] * c["dim"], c["heads"] * c["vdim"]
        return {"q": d.matrix(qk, H), "k": d.matrix(qk, H), "v": d.matrix(vv, H), "b": d.matrix(c["heads"], H),
                "a": d.matrix(c["heads"], H), "g": d.matrix(vv, H), "o": d.matrix(H, vv), "norm": d.normal(c["vdim"], std=0.1, mean=1.0),
                "A_log": torch.log(d.uniform(c["heads"], lo=1.0, hi=16.0, dtype=torch.float32)).to(BF16), "dt_bias": d.steps(c["heads"]),
                "q.conv": d.taps(qk, c["conv"]), "k.conv": d.taps(qk, c["conv"]), "v.conv": d.taps(vv, c["conv"])}
    if c["path"] == "ssm":
        inner = c["heads"] * c["vdim"]
        ch = inner + 2 * c["groups"] * c["state"]
        return {"in": d.matrix(inner + ch + c["heads"], H), "conv": d.taps(ch, c["conv"]), "conv.b": d.normal(ch, std=0.1),
                "dt_bias": d.steps(c["heads"]), "A_log": torch.log(d.uniform(c["heads"], lo=1.0, hi=16.0, dtype=torch.float32)).to(BF16),
                "D": d.normal(c["heads"], std=0.1, mean=1.0), "norm": d.normal(inner, std=0.1, mean=1.0), "o": d.matrix(H, inner)}
    if c["path"] == "scan":
        I, n = c["inner"], c["state"]
        return {"in": d.matrix(2 * I, H), "conv": d.taps(I, c["conv"]), "conv.b": d.normal(I, std=0.1), "x": d.matrix(c["rank"] + 2 * n, I),
                "dt": d.normal(I, c["rank"], std=0.3 * c["rank"] ** -0.5), "dt.b": d.steps(I),
                "A_log": torch.log(torch.arange(1, n + 1, device="cuda", dtype=torch.float32)).repeat(I, 1).to(BF16),
                "D": d.normal(I, std=0.1, mean=1.0), "o": d.matrix(H, I)}
    if c["path"] == "retention":
        qk, vv = c["heads"] * c["dim"], c["heads"] * c["vdim"]
        return {"q": d.matrix(qk, H), "k": d.matrix(qk, H), "v": d.matrix(vv, H), "g": d.matrix(vv, H), "o": d.matrix(H, vv)}
    E, F = c["experts"], c["ff"]
    names = ("up", "down") if c["kind"] == "relu2" else ("gate", "up", "down")
    w = {"router": d.matrix(E + (1 if c["kind"] == "relu2" else 0), H)}
    for p in [f"e{e}." for e in range(E)] + ([] if c["kind"] == "clamped" else ["shared."]):
        for n in names:
            w[p + n] = d.matrix(H, F) if n == "down" else d.matrix(F, H)
    if c["kind"] == "weigh_input":
        w["shared.sg"] = d.matrix(1, H)
    if c["kind"] == "relu2":
        w["correction"] = d.normal(E + 1, std=0.02)
    return w


def _slopes_decay(heads):
    """Retention's fixed decays: from 1 - 2^-5 to 1 - 2^-13 over the heads, evenly over the logarithm."""
    return [1.0 - 2.0 ** (-5.0 - 8.0 * h / max(1, heads - 1)) for h in range(heads)]


def _part(c):
    from gollmgo_b200.parts import PartSpec
    H = c["hidden"]
    if c["path"] == "attention":
        p = dict(hidden_size=H, num_heads=c["heads"], num_kv_heads=c["kv"], head_dim=c["dim"], window=c["window"] or None,
                 position=PartSpec("rope", dict(head_dim=c["dim"], rotary_dim=c["rot"], theta=500000.0)) if c["rot"] else PartSpec("none"))
        if c["softcap"]:
            p["softcap"] = c["softcap"]
        if c["sloped"]:
            p.update(distance_bias=True, sink=True, temperature=(0.1, 1024))
        return PartSpec("attention", p)
    if c["path"] == "delta":
        return PartSpec("gated_delta", dict(hidden_size=H, num_heads=c["heads"], num_kv_heads=c["kv"], head_dim=c["dim"],
                                            v_head_dim=c["vdim"], conv=c["conv"], eps=EPS))
    if c["path"] == "ssm":
        return PartSpec("mamba2", dict(hidden_size=H, num_heads=c["heads"], v_head_dim=c["vdim"], state=c["state"], groups=c["groups"],
                                       conv=c["conv"], norm_groups=c["groups"], eps=EPS))
    if c["path"] == "scan":
        return PartSpec("mamba1", dict(hidden_size=H, inner=c["inner"], state=c["state"], dt_rank=c["rank"], conv=c["conv"]))
    if c["path"] == "retention":
        return PartSpec("retention", dict(hidden_size=H, num_heads=c["heads"], head_dim=c["dim"], v_head_dim=c["vdim"],
                                          decay=_slopes_decay(c["heads"]), eps=EPS,
                                          position=PartSpec("rope", dict(head_dim=c["dim"], theta=10000.0))))
    p = dict(hidden_size=H, intermediate_size=c["ff"], experts=c["experts"], top=c["top"], router_bias=False)
    gated = ("gate", "up", "down")
    if c["kind"] == "clamped":
        p.update(router_weigh="softmax_all", groups=(4, 2), activation="clamped_swish", limit=7.0)
    elif c["kind"] == "weigh_input":
        p.update(router_weigh="sigmoid", weigh_input=True, shared_gate=True,
                 shared=PartSpec("gated_mlp", dict(hidden_size=H, intermediate_size=c["ff"], activation="silu", names=gated)))
    else:
        p.update(router_weigh="softmax_all", gated=False, activation="relu2", router_scale=2.5, correction=True, identity=1,
                 shared=PartSpec("mlp", dict(hidden_size=H, intermediate_size=c["ff"], activation="relu2", names=("up", "down"))))
    return PartSpec("moe", p)


def _state_shapes(c):
    if c["path"] == "delta":
        return [(c["heads"], c["vdim"], c["dim"]), (c["conv"] - 1, 2 * c["kv"] * c["dim"] + c["heads"] * c["vdim"])]
    if c["path"] == "ssm":
        return [(c["heads"], c["vdim"], c["state"]), (c["conv"] - 1, c["heads"] * c["vdim"] + 2 * c["groups"] * c["state"])]
    if c["path"] == "scan":
        return [(c["inner"], c["state"]), (c["conv"] - 1, c["inner"])]
    return [(c["heads"], c["vdim"], c["dim"])]


def _new_lens(c):
    if c["path"] == "moe":
        return [c["tokens"]]
    if c["path"] in ("attention", "model") and c["new"] == 1:
        return [1] * c["seqs"]
    return _lens(c["new"], c["seqs"])


def _decodes(c):
    return c["tokens"] <= 64 if c["path"] == "moe" else max(_new_lens(c)) == 1


def _inputs(c, seed):
    """The layer's input rows and, where earlier steps left something, what they left."""
    d = _Draws(seed, "inputs")
    lens = _new_lens(c)
    x = d.normal(sum(lens), c["hidden"])
    if c["path"] == "attention" and c["new"] == 1:
        return x, [(d.normal(n, c["kv"], c["dim"]), d.normal(n, c["kv"], c["dim"])) for n in _contexts(c)]
    if c["path"] in ("delta", "ssm", "scan", "retention") and _decodes(c):
        return x, [d.normal(len(lens), *s, std=0.3, dtype=torch.float32) for s in _state_shapes(c)]
    return x, None


def _captured(fn):
    """``fn`` as a captured step: warmed up on a side stream, captured, and what it returned."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = fn()
    return g, out


def _llama(c):
    return dict(architectures=["LlamaForCausalLM"], hidden_act="silu", rms_norm_eps=1e-5, num_hidden_layers=c["layers"],
                hidden_size=c["hidden"], num_attention_heads=c["heads"], num_key_value_heads=c["kv"], head_dim=c["dim"],
                intermediate_size=c["ff"], vocab_size=c["vocab"], rope_theta=500000.0, tie_word_embeddings=False,
                max_position_embeddings=32768)


def _prompts(c, seed):
    """Token ids: per sequence those of its context and the new ones."""
    g = torch.Generator().manual_seed(seed)
    ctx = _contexts(c) if c["new"] == 1 else [0] * c["seqs"]
    return [(torch.randint(0, c["vocab"], (n,), generator=g).tolist(), torch.randint(0, c["vocab"], (m,), generator=g).tolist())
            for n, m in zip(ctx, _new_lens(c))]


def _prepare_model(c, seed):
    from gollmgo_b200 import EngineConfig
    from gollmgo_b200.engine import ModelRunner, StepEntry
    seqs = _prompts(c, seed)
    longest = max(len(a) + len(b) for a, b in seqs)
    runner = ModelRunner(_llama(c), EngineConfig(
        dtype="bfloat16", block_size=PAGE, num_blocks=len(seqs) * (-(-longest // PAGE) + 1) + 8, max_batch_size=max(8, len(seqs)),
        max_token_budget=max(2048, c["new"] + 8), max_model_len=longest + 64), weights_seed=seed)
    entries = []
    for i, (ctx, new) in enumerate(seqs):
        if ctx:
            runner.step([StepEntry(i, ctx, [])])
        entries.append(StepEntry(i, new, [0] if c["new"] == 1 else [len(new) - 1]))
    return dict(path="model", runner=runner, entries=entries, keep=[len(a) for a, _ in seqs])


def _prepare_sample(c, seed):
    from gollmgo_b200 import SamplingParams
    from gollmgo_b200.sampling import Sampler
    R = c["rows"]
    logits = _Draws(seed, "logits").normal(R, c["vocab"], std=2.5, dtype=torch.float32)
    params = [SamplingParams(temperature=0.6 + 0.1 * (r % 5), top_k=(0, 50, 400)[r % 3], top_p=(0.9, 0.95, 0.0, 0.8)[r % 4],
                             seed=seed + r) for r in range(R)]
    return dict(path="sample", sampler=Sampler("cuda", R), logits=logits, params=params, draws=[(7 * r) % 100 for r in range(R)])


def prepare(case, seed):
    c = case
    if c["path"] == "model":
        return _prepare_model(c, seed)
    if c["path"] == "sample":
        return _prepare_sample(c, seed)
    from gollmgo_b200 import parts
    from gollmgo_b200.cache import CacheManager
    from gollmgo_b200.engine import BatchBuilder, StepEntry
    parts.set_matmul_precision()
    w = _weights(c, seed)
    x, before = _inputs(c, seed)
    lens = _new_lens(c)
    ctx = parts.BuildContext(BF16, "cuda", max_tokens=max(64, sum(lens)), max_seqs=max(8, len(lens)), page_size=PAGE)
    if c["path"] == "moe":
        part = parts.build_feed_forward(_part(c), ctx)
        part.load(w.__getitem__)
        call = lambda: part.forward(x, None)  # noqa: E731
        kept = ()
    else:
        part = parts.build_mixer(_part(c), ctx)
        part.load(w.__getitem__)
        need = part.cache_need()
        held = _contexts(c) if c["path"] == "attention" and c["new"] == 1 else [40 if before is not None else 0] * len(lens)
        pages = sum(-(-(h + n) // PAGE) for h, n in zip(held, lens)) + 1
        cm = CacheManager([need], PAGE, pages, len(lens), dtype=BF16, device="cuda")
        bb = BatchBuilder(cm, "cuda", query_tiles=getattr(part, "query_tiles", lambda: ())())
        view = cm.cache_view(0, need)
        for i, h in enumerate(held):
            cm.admit(i)
            if h:
                cm.append(i, h)
        if c["path"] == "attention":
            kept = view[:2]
            for t in kept:
                t.zero_()
            for i, (k, v) in enumerate(before or ()):
                n = k.shape[0]
                for t, rows in zip(kept, (k, v)):
                    full = torch.zeros(-(-n // PAGE) * PAGE, *rows.shape[1:], dtype=BF16, device="cuda")
                    full[:n] = rows
                    blocks = full.view(-1, PAGE, c["kv"], c["dim"]).transpose(1, 2)
                    table = torch.tensor(cm.block_table(i, 0)[:blocks.shape[0]], device="cuda")
                    t[table[table >= 0]] = blocks[table >= 0]
        else:
            kept = view if isinstance(view, tuple) else (view,)
            for t, start in zip(kept, before or ()):
                t.copy_(start)
        batch = bb.build([StepEntry(i, [0] * n, [0]) for i, n in enumerate(lens)])
        call = lambda: part.forward(x, batch, view)  # noqa: E731
    state = dict(path=c["path"], call=call, kept=kept, hold=(part, w, x))
    if _decodes(c):
        graph, y = _captured(call)
        if before is not None and c["path"] != "attention":
            for t, start in zip(kept, before):                 # the warm-up moved the recurrent state on
                t.copy_(start)
        state.update(graph=graph, y=y)
    return state


def run(state):
    s = state
    if s["path"] == "model":
        runner = s["runner"]
        logits = runner.step(s["entries"])
        for e, n in zip(s["entries"], s["keep"]):              # give the step's cache room back: the next pass is the same step
            if n:
                runner.cache.rollback(e.request_id, n)
            else:
                runner.release(e.request_id)
        return {"logits": logits}
    if s["path"] == "sample":
        s["sampler"].sample_async(s["logits"], s["params"], s["draws"])
        return {"tokens": s["sampler"].tokens}
    if "graph" in s:
        s["graph"].replay()
        y = s["y"]
    else:
        y = s["call"]()
    return {"y": y, **{f"kept{i}": t for i, t in enumerate(s["kept"])}}


# ---------------------------------------------------------------- what a pass cannot do without
def _pairs(c):
    """(query, key) pairs that attend."""
    win = c.get("window") or 1 << 40
    if c["new"] == 1:
        return sum(min(n + 1, win) for n in _contexts(c))
    return sum(sum(min(i + 1, win) for i in range(n)) for n in _new_lens(c))


def work(case):
    c = case
    if c["path"] == "sample":
        return {"bytes": 4.0 * c["rows"] * c["vocab"], "flops": 0.0}
    T = sum(_new_lens(c))
    H = c["hidden"]
    if c["path"] in ("attention", "model"):
        q, kv = c["heads"] * c["dim"], c["kv"] * c["dim"]
        layer = (2 * q + 2 * kv) * H
        cached = 2 * kv * (sum(min(n, c.get("window") or n) for n in _contexts(c)) if c["new"] == 1 else 0)
        if c["path"] == "attention":
            return {"bytes": 2.0 * (layer + 2 * T * H + 2 * T * kv + cached), "flops": 2.0 * T * layer + 4.0 * q * _pairs(c)}
        layer += 3 * H * c["ff"]
        R = c["seqs"]
        return {"bytes": 2.0 * (c["layers"] * (layer + cached + 2 * T * kv) + c["vocab"] * H + T * H) + 4.0 * R * c["vocab"],
                "flops": c["layers"] * (2.0 * T * layer + 4.0 * q * _pairs(c)) + 2.0 * R * c["vocab"] * H}
    if c["path"] == "moe":
        per = (2 if c["kind"] == "relu2" else 3) * H * c["ff"]
        used = min(c["experts"], T * c["top"]) + (0 if c["kind"] == "clamped" else 1)
        return {"bytes": 2.0 * (used * per + 2 * T * H), "flops": 2.0 * T * (c["top"] + (0 if c["kind"] == "clamped" else 1)) * per}
    weights = {"delta": lambda: H * (2 * c["kv"] * c["dim"] + 3 * c["heads"] * c["vdim"]),
               "ssm": lambda: H * (3 * c["heads"] * c["vdim"] + 2 * c["groups"] * c["state"]),
               "scan": lambda: 3 * H * c["inner"] + c["inner"] * (2 * c["rank"] + 2 * c["state"]),
               "retention": lambda: H * c["heads"] * (2 * c["dim"] + 3 * c["vdim"])}[c["path"]]()
    per_token = {"delta": lambda: 7 * c["heads"] * c["dim"] * c["vdim"], "ssm": lambda: 5 * c["heads"] * c["vdim"] * c["state"],
                 "scan": lambda: 6 * c["inner"] * c["state"], "retention": lambda: 5 * c["heads"] * c["dim"] * c["vdim"]}[c["path"]]()
    states = sum(math.prod(s) for s in _state_shapes(c)) * len(_new_lens(c)) * (2 if _decodes(c) else 1)
    return {"bytes": 2.0 * (weights + 2 * T * H) + 4.0 * states, "flops": 2.0 * T * weights + float(T * per_token)}


def tolerance(case):
    if case["path"] == "sample":
        return "exact"                  # whole numbers: a draw depends on its seed, its index and its row alone
    # bfloat16 activations between a layer's products: measured 2e-3 to 5e-3 from float64 for one layer and 1.8e-2 for the
    # logits behind four (two correct implementations differ by about 1.4 times that)
    return {"rel": 0.03, "max": 0.6} if case["path"] == "model" else {"rel": 0.012, "max": 0.3}


# ---------------------------------------------------------------- the same in float64
def _rms(x, eps=EPS):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, pos, rot, theta):
    """x [T, heads, size]: channel i of the first ``rot`` is paired with channel i + rot / 2."""
    if not rot:
        return x
    h = rot // 2
    ang = pos.to(F64)[:, None] * theta ** (-torch.arange(h, dtype=F64, device=x.device) * 2.0 / rot)[None, :]
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    u, v = x[..., :h], x[..., h:rot]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., rot:]], -1)


def _attend(q, k, v, first, c, sink=None):
    """q [n, heads, d] at positions first .. first + n, k and v [first + n, kv heads, d] -> [n, heads * d]."""
    n, nh, d = q.shape
    rep = nh // k.shape[1]
    i = torch.arange(first, first + n, device=q.device)[:, None]
    j = torch.arange(k.shape[0], device=q.device)[None, :]
    seen = j <= i
    if c.get("window"):
        seen = seen & (i - j < c["window"])
    out = torch.empty(n, nh, v.shape[-1], dtype=F64, device=q.device)
    for h in range(nh):
        s = (q[:, h] @ k[:, h // rep].T) * d ** -0.5
        if c.get("softcap"):
            s = c["softcap"] * torch.tanh(s / c["softcap"])
        if c.get("sloped"):
            s = s * (1.0 + 0.1 * torch.log(torch.floor((i + 1.0) / 1024) + 1.0)) - 2.0 ** (-8.0 * (h + 1) / nh) * (i - j)
        s = s.masked_fill(~seen, -math.inf)
        top = s.max(-1, keepdim=True).values
        e = torch.exp(s - top)
        z = e.sum(-1, keepdim=True)
        if sink is not None:
            z = z + torch.exp(sink[h] - top)
        out[:, h] = (e / z) @ v[:, h // rep]
    return out.reshape(n, -1)


def _exact_attention(c, x, before, w):
    lens, at, rows = _new_lens(c), 0, []
    for b, n in enumerate(lens):
        h = x[at:at + n]
        at += n
        first = before[b][0].shape[0] if before else 0
        pos = torch.arange(first, first + n, device=x.device)
        q, k, v = ((h @ w[m + "_proj.weight"].T).view(n, -1, c["dim"]) for m in "qkv")
        q, k = _rotate(q, pos, c["rot"], 500000.0), _rotate(k, pos, c["rot"], 500000.0)
        if before:
            k, v = torch.cat([before[b][0].double(), k]), torch.cat([before[b][1].double(), v])
        rows.append(_attend(q, k, v, first, c, w.get("sink")))
    return {"y": torch.cat(rows) @ w["o_proj.weight"].T, "kept0": None, "kept1": None}


def _conv(x, taps, carried, bias=None):
    """Causal convolution per channel; ``carried``: the inputs before the first row, oldest first -> (rows, the last inputs)."""
    n = taps.shape[1]
    full = torch.cat([carried, x])
    y = sum(full[j:j + x.shape[0]] * taps[:, j] for j in range(n))
    return _silu(y if bias is None else y + bias), full[full.shape[0] - (n - 1):]


def _recur(q, k, v, decay, S, beta=None):
    """S [H, d, dv] over the rows of q, k [T, H, d], v [T, H, dv], decay [T, H] -> (rows [T, H, dv], S)."""
    out = torch.empty_like(v)
    for t in range(v.shape[0]):
        S = S * decay[t][:, None, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out, S


def _exact_recurrent(c, x, before, w):
    lens, at, rows = _new_lens(c), 0, []
    states = [torch.zeros(len(lens), *s, dtype=F64, device=x.device) for s in _state_shapes(c)]
    if before:
        states = [b.double() for b in before]
    for b, n in enumerate(lens):
        h = x[at:at + n]
        at += n
        S = states[0][b].transpose(-1, -2) if c["path"] != "scan" else states[0][b]
        if c["path"] == "delta":
            H, G, d, dv = c["heads"], c["kv"], c["dim"], c["vdim"]
            qkv, last = _conv(h @ torch.cat([w["q"], w["k"], w["v"]]).T, torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]]), states[1][b])
            q, k, v = qkv[:, :G * d].view(n, G, d), qkv[:, G * d:2 * G * d].view(n, G, d), qkv[:, 2 * G * d:].view(n, H, dv)
            q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(H // G, 1)
            k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
            decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"]))
            o, S = _recur(q, k, v, decay, S, torch.sigmoid(h @ w["b"].T))
            o = (_rms(o) * w["norm"] * _silu(h @ w["g"].T).view(n, H, dv)).reshape(n, -1)
        elif c["path"] == "ssm":
            H, P, N, G = c["heads"], c["vdim"], c["state"], c["groups"]
            inner = H * P
            proj = h @ w["in"].T
            ch = inner + 2 * G * N
            mixed, last = _conv(proj[:, inner:inner + ch], w["conv"], states[1][b], w["conv.b"])
            xs = mixed[:, :inner].view(n, H, P)
            B, C = (mixed[:, inner + k * G * N:inner + (k + 1) * G * N].view(n, G, N).repeat_interleave(H // G, 1) for k in (0, 1))
            dt = torch.nn.functional.softplus(proj[:, inner + ch:] + w["dt_bias"])
            o, S = _recur(C, B, dt[:, :, None] * xs, torch.exp(-torch.exp(w["A_log"]) * dt), S)
            o = (o + w["D"][:, None] * xs).reshape(n, inner) * _silu(proj[:, :inner])
            o = _rms(o.view(n, G, -1)).view(n, inner) * w["norm"]
        elif c["path"] == "retention":
            H, d, dv = c["heads"], c["dim"], c["vdim"]
            pos = torch.arange(n, device=x.device) + (40 if before else 0)
            q, k = (_rotate((h @ w[m].T).view(n, H, d), pos, d, 10000.0) for m in "qk")
            g = torch.tensor(_slopes_decay(H), dtype=F64, device=x.device).expand(n, H)
            o, S = _recur(q, k * d ** -0.5, (h @ w["v"].T).view(n, H, dv), g, S)
            o, last = _rms(o).reshape(n, -1) * _silu(h @ w["g"].T), None
        else:
            I, N, R = c["inner"], c["state"], c["rank"]
            xz = h @ w["in"].T
            xs, last = _conv(xz[:, :I], w["conv"], states[1][b], w["conv.b"])
            low = xs @ w["x"].T
            dt = torch.nn.functional.softplus(low[:, :R] @ w["dt"].T + w["dt.b"])
            A, o = -torch.exp(w["A_log"]), torch.empty(n, I, dtype=F64, device=x.device)
            for t in range(n):
                S = S * torch.exp(dt[t][:, None] * A) + (dt[t] * xs[t])[:, None] * low[t, R:R + N][None, :]
                o[t] = S @ low[t, R + N:]
            o = (o + w["D"] * xs) * _silu(xz[:, I:])
        states[0][b] = S.transpose(-1, -2) if c["path"] != "scan" else S
        if last is not None:
            states[1][b] = last
        rows.append(o)
    return {"y": torch.cat(rows) @ w["o"].T, **{f"kept{i}": s for i, s in enumerate(states)}}


def _exact_moe(c, x, w):
    E, top = c["experts"], c["top"]
    z = x @ w["router"].T
    gate = torch.ones(x.shape[0], 1, dtype=F64, device=x.device)
    if c["kind"] == "weigh_input":
        s = torch.sigmoid(z)
        idx = s.topk(top, -1).indices
        wgt = s.gather(1, idx)
        gate = torch.sigmoid(x @ w["shared.sg"].T)
    else:
        s = torch.softmax(z, -1)
        choice = s
        if c["kind"] == "clamped":
            best = s.view(-1, 4, E // 4).max(-1).values.topk(2, -1).indices
            keep = torch.zeros(x.shape[0], 4, dtype=torch.bool, device=x.device).scatter_(1, best, True)
            choice = s.masked_fill(~keep.repeat_interleave(E // 4, 1), -1.0)
        else:
            choice = s + w["correction"]
        idx = choice.topk(top, -1).indices
        wgt = s.gather(1, idx)
        wgt = wgt / (wgt.sum(-1, keepdim=True) + 1e-20) * (2.5 if c["kind"] == "relu2" else 1.0)

    def ff(h, p):
        up = h @ w[p + "up"].double().T
        if c["kind"] == "relu2":
            a = torch.relu(up) ** 2
        elif c["kind"] == "clamped":
            g = torch.clamp(h @ w[p + "gate"].double().T, max=7.0)
            a = g * torch.sigmoid(1.702 * g) * (torch.clamp(up, -7.0, 7.0) + 1.0)
        else:
            a = _silu(h @ w[p + "gate"].double().T) * up
        return a @ w[p + "down"].double().T

    out = torch.zeros_like(x)
    for e in range(E + (1 if c["kind"] == "relu2" else 0)):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        if len(t):
            f = wgt[t, j][:, None]
            y = f * x[t] if e >= E else ff(f * x[t], f"e{e}.") if c["kind"] == "weigh_input" else f * ff(x[t], f"e{e}.")
            out.index_add_(0, t, y)
    if c["kind"] != "clamped":
        out = out + gate * ff(x, "shared.")
    return {"y": out}


def _exact_model(c, seed):
    def get(name, *shape):
        """Weights as the engine draws them for a seed: by the tensor's name alone."""
        if len(shape) == 1:
            return torch.ones(shape, dtype=F64, device="cuda")
        g = torch.Generator(device="cuda")
        g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:8], "little") & ((1 << 63) - 1))
        return torch.empty(shape, dtype=BF16, device="cuda").normal_(0.0, 0.02, generator=g).double()

    H, d = c["hidden"], c["dim"]
    seqs = [torch.tensor(a + b, device="cuda") for a, b in _prompts(c, seed)]
    embed = get("model.embed_tokens.weight", c["vocab"], H)
    xs = [embed[s] for s in seqs]
    del embed
    for i in range(c["layers"]):
        p = f"model.layers.{i}."
        w = {m: get(p + f"self_attn.{m}_proj.weight", {"q": c["heads"], "k": c["kv"], "v": c["kv"]}[m] * d, H) for m in "qkv"}
        w["o"] = get(p + "self_attn.o_proj.weight", H, c["heads"] * d)
        for m in ("gate", "up"):
            w[m] = get(p + f"mlp.{m}_proj.weight", c["ff"], H)
        w["down"] = get(p + "mlp.down_proj.weight", H, c["ff"])
        for b, x in enumerate(xs):
            n = x.shape[0]
            pos = torch.arange(n, device="cuda")
            h = _rms(x, 1e-5)
            q, k, v = ((h @ w[m].T).view(n, -1, d) for m in "qkv")
            x = x + _attend(_rotate(q, pos, d, 500000.0), _rotate(k, pos, d, 500000.0), v, 0, {}) @ w["o"].T
            h = _rms(x, 1e-5)
            xs[b] = x + (_silu(h @ w["gate"].T) * (h @ w["up"].T)) @ w["down"].T
    last = torch.stack([x[-1] for x in xs])
    return {"logits": _rms(last, 1e-5) @ get("lm_head.weight", c["vocab"], H).T}


def exact(case, seed):
    c = case
    if c["path"] == "sample":
        return None
    if c["path"] == "model":
        return _exact_model(c, seed)
    w = _weights(c, seed)
    x, before = _inputs(c, seed)
    if c["path"] == "moe":
        return _exact_moe(c, x.double(), {k: v if k[0] == "e" or (k.startswith("shared.") and k != "shared.sg") else v.double() for k, v in w.items()})
    w = {k: v.double() for k, v in w.items()}
    return (_exact_attention if c["path"] == "attention" else _exact_recurrent)(c, x.double(), before, w)
