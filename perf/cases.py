"""What a program has this framework do, as measurable cases: whole steps of the engine's step function and single layers through
the parts that models are made of, over the range of sizes they meet in use.

A case is a dict with a ``kind``:

* ``step``: one call of ``ModelRunner.step`` on a Qwen3 shape with a few of its layers -- decoded tokens (replayed from a captured
  graph, as the engine does) or portions of prompts; returns the logits.
* ``attention``: the attention mixer of a Qwen3-8B layer on a mixed step: portions of prompts behind cached context.
* ``experts``: the routed feed-forward with a shared expert of a Nogelorn layer.
* ``delta``: the gated delta rule (Senadra's form, a decay per channel; Ferodra's, one per head) on portions of prompts.
* ``latent``: attention over a cached latent (Galodra) on decoded tokens or portions of prompts.
* ``sample``: ``Sampler.sample`` on a step's logits with the usual mix of request parameters.

Weights are N(0, 0.02) as a freshly initialised model's, norm weights near 1; cached keys and values and layer inputs are N(0, 1), the
scale that norms leave.  Everything follows from the seed."""
import math
import zlib

import torch

DEV = "cuda"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DTYPES = {"bfloat16": BF16, "float32": F32}


# ---- the sizes -----------------------------------------------------------------------------------------------------
QWEN3 = {
    "0.6b": dict(vocab_size=151936, hidden_size=1024, intermediate_size=3072, num_attention_heads=16, num_key_value_heads=8, head_dim=128,
                 rms_norm_eps=1e-6, rope_theta=1000000.0, max_position_embeddings=40960, tie_word_embeddings=True),
    "8b": dict(vocab_size=151936, hidden_size=4096, intermediate_size=12288, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
               rms_norm_eps=1e-6, rope_theta=1000000.0, max_position_embeddings=40960, tie_word_embeddings=False),
}
EXPERTS = {  # one layer with routed experts and a shared one
    "2k": dict(width=2048, heads=16, experts=64, top=5, ff=1408),
    "4k": dict(width=4096, heads=32, experts=64, top=5, ff=2048),
}
DELTA = {
    "channel-2k": dict(width=2048, heads=16, kv_heads=8, dim=128, vdim=128, conv=4, rank=64),
    "head-2k": dict(width=2048, heads=16, kv_heads=8, dim=128, vdim=128, conv=4, rank=0),
    "channel-4k": dict(width=4096, heads=32, kv_heads=16, dim=128, vdim=128, conv=4, rank=64),
}
LATENT = {
    "2k": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, rank=512),
    "4k": dict(width=4096, heads=32, dim=128, rot=64, vdim=128, rank=512),
}
EPS = 1e-6


def listed():
    return [
        # one user's chat on the small model: the shortest step there is, bound by launches and latency
        dict(name="decode_one", kind="step", shape="0.6b", layers=8, dtype="bfloat16", seqs=1, tokens=1, ctx_lo=90, ctx_hi=90),
        # the benchmark's own point: eight requests behind prompts of 1,024 tokens
        dict(name="decode_eight", kind="step", shape="8b", layers=4, dtype="bfloat16", seqs=8, tokens=1, ctx_lo=1024, ctx_hi=1056),
        # a loaded server: many requests of all lengths
        dict(name="decode_many", kind="step", shape="8b", layers=4, dtype="bfloat16", seqs=61, tokens=1, ctx_lo=100, ctx_hi=2100),
        # one long prompt as one step
        dict(name="prompt", kind="step", shape="8b", layers=4, dtype="bfloat16", seqs=1, tokens=2048, ctx_lo=0, ctx_hi=0),
        # chunked prefill: later portions of several prompts in one step
        dict(name="attention_chunks", kind="attention", shape="8b", seqs=3, tokens=1361, ctx_lo=200, ctx_hi=6000),
        dict(name="experts_prompt", kind="experts", shape="2k", tokens=2048),
        # a decode step of a small batch through the experts
        dict(name="experts_few", kind="experts", shape="2k", tokens=24),
        dict(name="delta_prompt", kind="delta", shape="channel-2k", seqs=1, tokens=1500),
        dict(name="latent_decode", kind="latent", shape="2k", seqs=48, tokens=48, ctx_lo=800, ctx_hi=4000),
        dict(name="latent_prompt", kind="latent", shape="2k", seqs=2, tokens=1337, ctx_lo=0, ctx_hi=600),
        # the true 32-bit path, which results are checked against
        dict(name="float32_prompt", kind="step", shape="0.6b", layers=2, dtype="float32", seqs=2, tokens=301, ctx_lo=0, ctx_hi=40),
        # the end of every step of a server whose users sample
        dict(name="sample", kind="sample", rows=48, vocab=151936),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "prompt", "float32", "attention", "experts", "delta", "latent", "sample"])
    if kind == "decode":
        hi = _log(rng, 60, 4000)
        return dict(kind="step", shape=rng.choice(["0.6b", "8b"]), layers=rng.randint(2, 4), dtype="bfloat16", seqs=_log(rng, 1, 64),
                    tokens=1, ctx_lo=max(1, hi // rng.randint(1, 8)), ctx_hi=hi)
    if kind == "prompt":
        n = rng.randint(1, 4)
        hi = rng.choice([0, _log(rng, 30, 2000)])
        return dict(kind="step", shape=rng.choice(["0.6b", "8b"]), layers=rng.randint(2, 4), dtype="bfloat16", seqs=n, tokens=_log(rng, 2 * n, 2048),
                    ctx_lo=hi // 3, ctx_hi=hi)
    if kind == "float32":
        n = rng.randint(1, 4)
        hi = _log(rng, 10, 300)
        decode = rng.random() < 0.4
        return dict(kind="step", shape="0.6b", layers=rng.randint(1, 3), dtype="float32", seqs=n, tokens=1 if decode else _log(rng, 2 * n, 400),
                    ctx_lo=hi // 2, ctx_hi=hi)
    if kind == "attention":
        n = rng.randint(1, 6)
        hi = _log(rng, 50, 7000)
        return dict(kind="attention", shape=rng.choice(["0.6b", "8b"]), seqs=n, tokens=_log(rng, 40 * n, 2048), ctx_lo=hi // 5, ctx_hi=hi)
    if kind == "experts":
        return dict(kind="experts", shape=rng.choice(["2k", "4k"]), tokens=_log(rng, 1, 2048))
    if kind == "delta":
        n = rng.randint(1, 4)
        return dict(kind="delta", shape=rng.choice(sorted(DELTA)), seqs=n, tokens=_log(rng, 8 * n, 2048))
    if kind == "latent":
        n = _log(rng, 1, 64)
        hi = _log(rng, 40, 4000)
        if rng.random() < 0.5:
            return dict(kind="latent", shape=rng.choice(["2k", "4k"]), seqs=n, tokens=n, ctx_lo=hi // 4, ctx_hi=hi)
        n = rng.randint(1, 4)
        return dict(kind="latent", shape="2k", seqs=n, tokens=_log(rng, 8 * n, 1400), ctx_lo=0, ctx_hi=_log(rng, 40, 1000))
    return dict(kind="sample", rows=_log(rng, 1, 64), vocab=rng.choice([32768, 50257, 151936]))


# ---- inputs from a seed ------------------------------------------------------------------------------------------------
def _gen(seed, name):
    return torch.Generator(DEV).manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)


def _normal(seed, name, shape, std=1.0, dtype=BF16):
    return (torch.randn(shape, generator=_gen(seed, name), device=DEV, dtype=F32) * std).to(dtype)


def _uniform(seed, name, shape, lo, hi, dtype=F32):
    return (torch.rand(shape, generator=_gen(seed, name), device=DEV, dtype=F32) * (hi - lo) + lo).to(dtype)


def _tensor(seed, name, shape, dtype=BF16):
    """Tensor ``name`` of the model: what a file would hold (16 bits; a recurrence's own numbers as such layers are initialised)."""
    shape = tuple(shape)
    if name.endswith("A_log"):
        return torch.log(_uniform(seed, name, shape, 1.0, 16.0)).to(dtype)
    if name.endswith("dt_bias"):
        dt = torch.exp(_uniform(seed, name, shape, math.log(1e-3), math.log(1e-1)))
        return torch.log(torch.expm1(dt)).to(dtype)
    if name.endswith(".conv"):
        return _uniform(seed, name, shape, -0.5, 0.5, dtype)
    if "norm" in name:
        return _uniform(seed, name, shape, 0.9, 1.1, dtype)
    return _normal(seed, name, shape, 0.02, dtype)


def _ints(seed, name, n, lo, hi):
    return torch.randint(lo, hi, (n,), generator=torch.Generator().manual_seed((int(seed) * 7919 + zlib.crc32(name.encode())) & 0x7FFFFFFF)).tolist()


def _contexts(case):
    """The cached tokens of each sequence: spread evenly from ctx_lo to ctx_hi, long and short ones side by side."""
    n, lo, hi = case["seqs"], case["ctx_lo"], case["ctx_hi"]
    return [lo + ((i * 37) % n) * (hi - lo) // max(1, n - 1) if n > 1 else hi for i in range(n)]


def _portions(case):
    """How many tokens each sequence brings: ``tokens`` in all (one each when decoding), in uneven shares."""
    n, total = case["seqs"], case["tokens"]
    if total <= n:
        return [1] * n
    shares = [1.0 + 2.0 * ((i * 5) % n) for i in range(n)]
    out = [max(1, int(total * s / sum(shares))) for s in shares]
    out[-1] = max(1, out[-1] + total - sum(out))
    return out


# ---- models and steps --------------------------------------------------------------------------------------------------
def _model(arch, config, seed, dtype):
    from iian_b200.config.registry import get_architecture
    from iian_b200.engine.model import Model
    from iian_b200.weights.loader import WeightSource

    class Given(WeightSource):
        def describe(self):
            return "drawn"

        def check(self, declared):
            pass

        def has(self, name):
            return not name.endswith("proj.bias")

        def fetch(self, name, spec, compute, device):
            return _tensor(seed, name, spec.shape).to(compute)

    a = get_architecture(arch)
    return Model(a, a.load_config(config), dtype, DEV, Given())


def _requests(model, case, dtype, seed, vocab):
    """A runner whose cache holds each sequence's context, and the entries of the step: (runner, entries)."""
    from iian_b200.engine.runner import ModelRunner, StepEntry
    ctxs, news = _contexts(case) if "ctx_lo" in case else [0] * case["seqs"], _portions(case)
    capacity = sum(-(-(c + n) // 16) * 16 for c, n in zip(ctxs, news)) + 64
    runner = ModelRunner(model, block_size=16, capacity_tokens=capacity, max_num_seqs=max(8, case["seqs"]), cuda_graphs=True,
                         max_model_len=max(c + n for c, n in zip(ctxs, news)) + 16)
    mgr, entries = runner.manager, []
    tokens = _ints(seed, "tokens", sum(news), 5, vocab - 5)
    for i, (c, n) in enumerate(zip(ctxs, news)):
        rc = mgr.new_request()
        mgr.allot_state(rc)
        if not mgr.allocate(rc, 0, c + n):
            raise RuntimeError("the cache is too small")
        at = sum(news[:i])
        entries.append(StepEntry(rc, tokens[at: at + n], c, [n - 1]))
    return runner, entries


def _kept(seed, layer, i, heads, ctx, dim, dtype):
    """Cached keys and values of a sequence: [ctx, heads, dim] each."""
    return tuple(_normal(seed, "%s %d %d" % (w, layer, i), (ctx, heads, dim), 1.0).to(dtype) for w in "kv")


def _fill(runner, entries, seed, layers, heads, dim, dtype):
    for layer in range(layers):
        view = runner.storage.view(layer)
        for i, e in enumerate(entries):
            if not e.start:
                continue
            k, v = _kept(seed, layer, i, heads, e.start, dim, dtype)
            pages = -(-e.start // 16)
            table = torch.tensor(list(e.cache.tables[view.group])[:pages], device=DEV, dtype=torch.long)
            for t, cells in ((k, view.k), (v, view.v)):
                full = torch.zeros(pages * 16, heads, dim, device=DEV, dtype=dtype)
                full[: e.start] = t
                cells[table] = full.view(pages, 16, heads, dim).transpose(1, 2)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        cfg, dtype = QWEN3[case["shape"]], DTYPES[case["dtype"]]
        model = _model("Qwen3ForCausalLM", dict(cfg, num_hidden_layers=case["layers"]), seed, case["dtype"])
        runner, entries = _requests(model, case, dtype, seed, cfg["vocab_size"])
        _fill(runner, entries, seed, case["layers"], cfg["num_key_value_heads"], cfg["head_dim"], dtype)
        runner.step(entries)  # an engine warms up before it serves: graphs are captured, workspaces sized
        return dict(kind=kind, runner=runner, entries=entries)
    if kind == "attention":
        cfg = dict(QWEN3[case["shape"]], vocab_size=256, intermediate_size=256)
        model = _model("Qwen3ForCausalLM", dict(cfg, num_hidden_layers=1), seed, "bfloat16")
        runner, entries = _requests(model, case, BF16, seed, 256)
        _fill(runner, entries, seed, 1, cfg["num_key_value_heads"], cfg["head_dim"], BF16)
        view = runner.storage.view(0)
    elif kind == "experts":
        s = EXPERTS[case["shape"]]
        att = {"heads": s["heads"], "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
        mlp = {"kind": "moe", "expert": {"ff": s["ff"]}, "router": {"experts": s["experts"], "top": s["top"]}, "shared": {"ff": s["ff"]}}
        model = _model("Nogelorn", {"architecture": "Nogelorn", "vocab": 256, "width": s["width"], "norm": {"eps": EPS},
                                    "layers": [{"type": "attention", "mixer": att, "mlp": mlp}]}, seed, "bfloat16")
        runner, entries = _requests(model, dict(seqs=1, tokens=case["tokens"]), BF16, seed, 256)
        view = None
    elif kind == "delta":
        s = DELTA[case["shape"]]
        mixer = {k: s[k] for k in ("heads", "kv_heads", "dim", "vdim", "conv")}
        if s["rank"]:
            model = _model("Senadra", {"architecture": "Senadra", "vocab": 256, "width": s["width"], "norm": {"eps": EPS}, "layers": [
                {"type": "channel_delta", "mixer": dict(mixer, decay_rank=s["rank"], gate_rank=s["rank"]), "mlp": None}]}, seed, "bfloat16")
        else:
            model = _model("Ferodra", {"architecture": "Ferodra", "vocab": 256, "width": s["width"], "norm": {"eps": EPS}, "layers": [
                {"type": "delta", "mixer": mixer, "mlp": None}]}, seed, "bfloat16")
        runner, entries = _requests(model, case, BF16, seed, 256)
        view = runner.storage.view(0)
    elif kind == "latent":
        s = LATENT[case["shape"]]
        mixer = {"heads": s["heads"], "dim": s["dim"], "rot_dim": s["rot"], "vdim": s["vdim"], "kv_rank": s["rank"],
                 "scale": (s["dim"] + s["rot"]) ** -0.5, "rot": {"dims": s["rot"], "base": 10000.0}, "mask": {"size": 4096}}
        model = _model("Galodra", {"architecture": "Galodra", "vocab": 256, "width": s["width"], "norm": {"eps": EPS}, "postln_alpha": 2.0,
                                   "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": None}]}, seed, "bfloat16")
        runner, entries = _requests(model, case, BF16, seed, 256)
        view = runner.storage.view(0)
        for i, e in enumerate(entries):
            if e.start:
                pages = -(-e.start // 16)
                table = torch.tensor(list(e.cache.tables[view.group])[:pages], device=DEV, dtype=torch.long)
                full = torch.zeros(pages * 16, s["rank"] + s["rot"], device=DEV, dtype=BF16)
                full[: e.start] = _normal(seed, "rows %d" % i, (e.start, s["rank"] + s["rot"]))
                view.rows[table] = full.view(pages, 16, -1)
    else:
        return dict(kind=kind, **_sampling(case, seed))
    ctx = runner.build_context(entries)
    block = model.blocks[0]
    x = _normal(seed, "x", (ctx.num_tokens, model.hidden_size))
    return dict(kind=kind, runner=runner, entries=entries, ctx=ctx, x=x, view=view, part=block.feed_forward if kind == "experts" else block.mixer)


def _sampling(case, seed):
    from iian_b200.sampling.params import SamplingParams
    from iian_b200.sampling.sampler import Sampler
    rows = case["rows"]
    # a model's logits: a broad bell with a few likely tokens far out
    logits = _normal(seed, "logits", (rows, case["vocab"]), 2.0, F32)
    logits += 4.0 * _normal(seed, "likely", (rows, case["vocab"]), 1.0, F32).clamp_min(3.0).sub_(3.0)
    params = [SamplingParams(**p) for p in _settings(rows)]
    return dict(sampler=Sampler(logits.device), logits=logits, params=params, seeds=[int(seed) * 1000 + i for i in range(rows)],
                indices=[(i * 13) % 200 for i in range(rows)])


def _settings(rows):
    usual = [dict(temperature=0.7, top_p=0.8, top_k=20), dict(temperature=0.6, top_p=0.95, top_k=20), dict(temperature=1.0),
             dict(temperature=0.8, top_p=0.9), dict(temperature=1.0, min_p=0.05), dict(temperature=0.0), dict(temperature=0.7, top_k=50)]
    return [usual[i % len(usual)] for i in range(rows)]


def run(state):
    kind = state["kind"]
    if kind == "step":
        return state["runner"].step(state["entries"]).clone()  # the step's own logits live in the runner, until its next step
    if kind == "sample":
        return torch.tensor(state["sampler"].sample(state["logits"], state["params"], state["seeds"], state["indices"]))
    if kind == "experts":
        return state["part"].forward(state["x"], state["ctx"])
    if kind == "delta":
        state["view"].state.zero_()  # new requests start from nothing
        return {"out": state["part"].forward(state["x"], state["ctx"], state["view"], True), "state": state["view"].state}
    return state["part"].forward(state["x"], state["ctx"], state["view"], True)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 0.0}
    if kind in ("step", "attention"):
        c = QWEN3[case["shape"]]
        ctxs, news = _contexts(case), _portions(case)
        n, e = sum(news), 4 if case.get("dtype") == "float32" else 2
        q, kv, h = c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"], c["hidden_size"]
        w = h * (q + 2 * kv) + q * h + (3 * h * c["intermediate_size"] if kind == "step" else 0)
        pairs = sum(t * p + t * (t + 1) / 2 for p, t in zip(ctxs, news))
        layers = case["layers"] if kind == "step" else 1
        cached = sum(p + t for p, t in zip(ctxs, news))
        by = layers * e * (w + 2 * kv * cached + 2 * kv * n) + (0 if kind == "step" else 2 * e * n * h)
        fl = layers * (2.0 * n * w + 4.0 * q * pairs)
        if kind == "step":
            by += e * c["vocab_size"] * h + len(news) * c["vocab_size"] * 4 + n * h * e
            fl += 2.0 * len(news) * c["vocab_size"] * h
        return {"bytes": float(by), "flops": fl}
    if kind == "experts":
        s, n = EXPERTS[case["shape"]], case["tokens"]
        reached = s["experts"] * (1.0 - (1.0 - s["top"] / s["experts"]) ** n)
        one = 3 * s["width"] * s["ff"]
        return {"bytes": 2.0 * ((reached + 1) * one + s["experts"] * s["width"] + 2 * n * s["width"]),
                "flops": 2.0 * n * ((s["top"] + 1) * one + s["experts"] * s["width"])}
    if kind == "delta":
        s, n = DELTA[case["shape"]], case["tokens"]
        qk, v = s["kv_heads"] * s["dim"], s["heads"] * s["vdim"]
        z = s["heads"] * s["dim"]
        low = s["rank"] * (2 * s["width"] + z + v) if s["rank"] else s["width"] * (s["heads"] + v)
        w = s["width"] * (2 * qk + v + s["heads"]) + low + s["width"] * v
        return {"bytes": 2.0 * (w + 2 * n * s["width"]) + 4.0 * 2 * case["seqs"] * s["heads"] * s["dim"] * s["vdim"],
                "flops": 2.0 * n * w + 6.0 * n * s["heads"] * s["dim"] * s["vdim"]}
    s = LATENT[case["shape"]]
    ctxs, news = _contexts(case), _portions(case)
    n, width = sum(news), s["rank"] + s["rot"]
    # every head scores the expanded keys and values (the cheaper form for long portions); the cached rows are read once
    w = s["width"] * (s["heads"] * (s["dim"] + s["rot"]) + width) + s["heads"] * (s["dim"] + s["vdim"]) * s["rank"] + s["heads"] * s["vdim"] * s["width"]
    pairs = sum(t * p + t * (t + 1) / 2 for p, t in zip(ctxs, news))
    return {"bytes": 2.0 * (w + width * (sum(ctxs) + 2 * n) + 2 * n * s["width"]),
            "flops": 2.0 * n * w + 2.0 * s["heads"] * (s["dim"] + s["rot"] + s["vdim"]) * pairs}


def tolerance(case):
    return TOLERANCE["float32" if case.get("dtype") == "float32" else case["kind"]]


# about four times the differences from ``exact`` (a whole step of 2 to 8 layers 0.011 to 0.014, single layers 0.0036 to 0.0042, the 32-bit
# step 3e-6, sampled tokens none; a draw may fall on the other side of a border between two tokens when sums are taken in another order)
TOLERANCE = {
    "step": {"rel": 0.05},
    "float32": {"rel": 1.2e-5},
    "attention": {"rel": 0.016},
    "experts": {"rel": 0.015},
    "delta": {"rel": 0.015},
    "latent": {"rel": 0.017},
    "sample": {"differ": 0.05},
}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------
def _rms(x, w, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _turn(x, pos, dims, base):
    """Rotation of the first ``dims`` entries of the last axis, entry i with entry i + dims / 2; x [N, heads, D]."""
    half = dims // 2
    f = pos.to(F64)[:, None] * base ** (-torch.arange(half, device=DEV, dtype=F64) * 2 / dims)
    c, s = torch.cos(f)[:, None], torch.sin(f)[:, None]
    a, b = x[..., :half], x[..., half: dims]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


def _attend(q, k, v, start, scale, sink=None, window=None):
    """q [t, H, D], k [c, H, D], v [c, H, E] (the keys from position 0): [t, H, E]."""
    t, c = q.shape[0], k.shape[0]
    at = torch.arange(start, start + t, device=DEV)[:, None]
    key = torch.arange(c, device=DEV)[None]
    hidden = (key > at) | (at - key >= (window or 1 << 30))
    out = torch.empty(t, q.shape[1], v.shape[2], device=DEV, dtype=F64)
    for h in range(q.shape[1]):
        z = (q[:, h] @ k[:, h].T * scale).masked_fill_(hidden, float("-inf"))
        if sink is not None:
            z = torch.cat([z, sink[h].expand(t, 1)], 1)
        out[:, h] = torch.softmax(z, -1)[:, :c] @ v[:, h]
    return out


def _qwen3_attention(x, c, seed, layer, ctxs, news, dtype):
    H, G, D, hid = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["hidden_size"]
    p = "model.layers.%d.self_attn." % layer
    W = lambda name, *shape: _tensor(seed, p + name + ".weight", shape).to(F64)  # noqa: E731
    q = _rms((x @ W("q_proj", H * D, hid).T).view(-1, H, D), W("q_norm", D))
    k = _rms((x @ W("k_proj", G * D, hid).T).view(-1, G, D), W("k_norm", D))
    v = (x @ W("v_proj", G * D, hid).T).view(-1, G, D)
    out, at = [], 0
    for i, (ctx, n) in enumerate(zip(ctxs, news)):
        pos = torch.arange(ctx, ctx + n, device=DEV)
        hk, hv = _kept(seed, layer, i, G, ctx, D, dtype)
        kk = torch.cat([hk.to(F64), _turn(k[at: at + n], pos, D, c["rope_theta"])]).repeat_interleave(H // G, 1)
        vv = torch.cat([hv.to(F64), v[at: at + n]]).repeat_interleave(H // G, 1)
        out.append(_attend(_turn(q[at: at + n], pos, D, c["rope_theta"]), kk, vv, ctx, D ** -0.5))
        at += n
    return torch.cat(out).view(-1, H * D) @ W("o_proj", hid, H * D).T


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return _exact_sample(case, seed)
    if kind == "step":
        c, dtype = QWEN3[case["shape"]], DTYPES[case["dtype"]]
        ctxs, news = _contexts(case), _portions(case)
        ids = torch.tensor(_ints(seed, "tokens", sum(news), 5, c["vocab_size"] - 5), device=DEV)
        embed = _tensor(seed, "model.embed_tokens.weight", (c["vocab_size"], c["hidden_size"]))
        x = embed[ids].to(F64)
        for layer in range(case["layers"]):
            p = "model.layers.%d." % layer
            W = lambda name, *shape: _tensor(seed, p + name + ".weight", shape).to(F64)  # noqa: E731
            x = x + _qwen3_attention(_rms(x, W("input_layernorm", c["hidden_size"])), c, seed, layer, ctxs, news, dtype)
            h = _rms(x, W("post_attention_layernorm", c["hidden_size"]))
            a = torch.nn.functional.silu(h @ W("mlp.gate_proj", c["intermediate_size"], c["hidden_size"]).T)
            a *= h @ W("mlp.up_proj", c["intermediate_size"], c["hidden_size"]).T
            x = x + a @ W("mlp.down_proj", c["hidden_size"], c["intermediate_size"]).T
        last = torch.cumsum(torch.tensor(news, device=DEV), 0) - 1
        x = _rms(x[last], _tensor(seed, "model.norm.weight", (c["hidden_size"],)).to(F64))
        head = embed if c["tie_word_embeddings"] else _tensor(seed, "lm_head.weight", (c["vocab_size"], c["hidden_size"]))
        return torch.cat([x @ w.to(F64).T for w in head.split(16384)], 1)
    if kind == "attention":
        c, ctxs, news = QWEN3[case["shape"]], _contexts(case), _portions(case)
        x = _normal(seed, "x", (sum(news), c["hidden_size"])).to(F64)
        return _qwen3_attention(x, c, seed, 0, ctxs, news, BF16)
    if kind == "experts":
        s = EXPERTS[case["shape"]]
        x = _normal(seed, "x", (case["tokens"], s["width"])).to(F64)
        W = lambda name, *shape: _tensor(seed, "l0.mlp." + name, shape).to(F64)  # noqa: E731
        score, chosen = torch.topk(x @ W("router", s["experts"], s["width"]).T + W("router.b", s["experts"]), s["top"], -1)
        weight = torch.softmax(score, -1)

        def one(name, u):
            act = torch.nn.functional.silu(u @ W(name + ".gate", s["ff"], s["width"]).T) * (u @ W(name + ".up", s["ff"], s["width"]).T)
            return act @ W(name + ".down", s["width"], s["ff"]).T

        out = one("shared", x)
        for e in range(s["experts"]):
            row, place = torch.nonzero(chosen == e, as_tuple=True)
            if len(row):
                out.index_add_(0, row, weight[row, place, None] * one("e%d" % e, x[row]))
        return out
    if kind == "delta":
        return _exact_delta(case, seed)
    s, ctxs, news = LATENT[case["shape"]], _contexts(case), _portions(case)
    H, D, R, V, K = s["heads"], s["dim"], s["rot"], s["vdim"], s["rank"]
    x = _normal(seed, "x", (sum(news), s["width"])).to(F64)
    W = lambda name, *shape: _tensor(seed, "l0.mix." + name, shape).to(F64)  # noqa: E731
    q = (x @ W("q", H * (D + R), s["width"]).T).view(-1, H, D + R)
    row = x @ W("dkv", K + R, s["width"]).T
    lat, kr = _rms(row[:, :K], W("dkv.norm", K)), row[:, None, K:]
    uk, uv, sink = W("uk", H * D, K).view(H, D, K), W("uv", H * V, K).view(H, V, K), W("sink", H)
    out, at = [], 0
    for i, (ctx, n) in enumerate(zip(ctxs, news)):
        pos = torch.arange(ctx, ctx + n, device=DEV)
        part = slice(at, at + n)
        old = _normal(seed, "rows %d" % i, (ctx, K + R)).to(F64) if ctx else torch.zeros(0, K + R, device=DEV, dtype=F64)
        rows = torch.cat([old, torch.cat([lat[part], _turn(kr[part], pos, R, 10000.0)[:, 0]], -1)])
        qq = torch.cat([torch.einsum("thd,hdk->thk", q[part, :, :D], uk), _turn(q[part, :, D:], pos, R, 10000.0)], -1)
        o = _attend(qq, rows[:, None].expand(-1, H, -1), rows[:, None, :K].expand(-1, H, -1), ctx, (D + R) ** -0.5, sink, 4096)
        out.append(torch.einsum("thk,hvk->thv", o, uv).reshape(n, H * V))
        at += n
    return torch.cat(out) @ W("o", s["width"], H * V).T


def _exact_delta(case, seed):
    s, news = DELTA[case["shape"]], _portions(case)
    H, G, D, V, hid, taps = s["heads"], s["kv_heads"], s["dim"], s["vdim"], s["width"], s["conv"]
    n = sum(news)
    x = _normal(seed, "x", (n, hid)).to(F64)
    W = lambda name, *shape: _tensor(seed, "l0.mix." + name, shape).to(F64)  # noqa: E731
    flow = torch.cat([x @ W("q", G * D, hid).T, x @ W("k", G * D, hid).T, x @ W("v", H * V, hid).T], 1)
    filt = torch.cat([W("q.conv", G * D, taps), W("k.conv", G * D, taps), W("v.conv", H * V, taps)])
    rate = torch.exp(W("A_log", H))
    if s["rank"]:
        z = x @ W("a1", s["rank"], hid).T @ W("a2", H * D, s["rank"]).T + W("dt_bias", H * D)
        g = torch.exp(-rate[:, None] * torch.nn.functional.softplus(z).view(n, H, D))
        gate = torch.sigmoid(x @ W("g1", s["rank"], hid).T @ W("g2", H * V, s["rank"]).T)
    else:
        z = x @ W("a", H, hid).T + W("dt_bias", H)
        g = torch.exp(-rate * torch.nn.functional.softplus(z))[..., None].expand(n, H, D)
        gate = torch.nn.functional.silu(x @ W("g", H * V, hid).T)
    beta = torch.sigmoid(x @ W("b", H, hid).T)
    heads, at = torch.empty(n, H, V, device=DEV, dtype=F64), 0
    for m in news:
        padded = torch.cat([torch.zeros(taps - 1, flow.shape[1], device=DEV, dtype=F64), flow[at: at + m]])
        act = torch.nn.functional.silu(sum(padded[j: j + m] * filt[:, j] for j in range(taps)))
        q, k, v = act[:, : G * D].view(m, G, D), act[:, G * D: 2 * G * D].view(m, G, D), act[:, 2 * G * D:].view(m, H, V)
        q = (q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * D ** -0.5).repeat_interleave(H // G, 1)
        k = (k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
        S = torch.zeros(H, D, V, device=DEV, dtype=F64)
        for t in range(m):
            S = S * g[at + t, :, :, None]
            u = beta[at + t, :, None] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
            S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
            heads[at + t] = torch.bmm(q[t, :, None], S)[:, 0]
        at += m
    normed = _rms(heads, W("norm", V)).reshape(n, H * V) * gate
    return {"out": normed @ W("o", hid, H * V).T, "state": None}


def _exact_sample(case, seed):
    """Temperature, min-p, top-k, top-p and the draw in vocabulary order, in 64 bits."""
    st = _sampling(case, seed)
    mask = (1 << 64) - 1

    def mix(v):
        v = (v + 0x9E3779B97F4A7C15) & mask
        v = ((v ^ (v >> 30)) * 0xBF58476D1CE4E5B9) & mask
        v = ((v ^ (v >> 27)) * 0x94D049BB133111EB) & mask
        return v ^ (v >> 31)

    out = []
    for r, p in enumerate(_settings(case["rows"])):
        row = st["logits"][r].to(F64)
        if p["temperature"] == 0.0:
            out.append(int(row.argmax()))
            continue
        z = row / p["temperature"]
        keep = torch.ones_like(z, dtype=torch.bool)
        if p.get("min_p"):
            keep &= z >= z.max() + math.log(p["min_p"])
        if p.get("top_k"):
            keep &= z >= torch.topk(z, p["top_k"]).values[-1]
        mass = torch.where(keep, torch.exp(z - z.max()), torch.zeros_like(z))
        if p.get("top_p", 1.0) < 1.0:
            ordered, place = torch.sort(mass, descending=True, stable=True)
            before = torch.cumsum(ordered, 0) - ordered
            mass[place[before >= p["top_p"] * mass.sum()]] = 0.0
        u = (mix(mix(st["seeds"][r] & mask) ^ ((st["indices"][r] * 0xD1B54A32D192ED03) & mask)) >> 40) / float(1 << 24)
        run = torch.cumsum(mass, 0)
        out.append(int(torch.searchsorted(run, u * run[-1], right=True)))
    return torch.tensor(out)
