"""The work that is measured: what users of this package have it do, through its public entry points.

    predict     DiffGPT.predict_samples: host frame in, host forecasts out (fp32 model, where launches and latency count)
    forward     Model.forward over a batch of whole sequences: scoring, perplexity, anomaly scores
    steps       StepRunner: requests whose tokens are given in portions and one by one, logits at the places asked for
    decode      DecodeRun, the loop under Engine.generate_many: `load` of new prompts, then every step.  `free` draws every
                token (Monte-Carlo futures); otherwise all tokens but the last are given beforehand (exogenous channels,
                back-tests), which makes the last step's logits a function of the inputs alone
    attention   ops.rope_qknorm_kvappend + ops.fmha_prefill, one layer's attention over long sequences

Models: the GPT of the package's four reference configurations (`GPTS`), and Delunex and Kipolix at the sizes of the
benchmark's design runs (`SIZES`), with random weights.  `exact` holds plain float64 restatements of the three models.
"""

import math

import numpy as np
import torch
import torch.nn.functional as F

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}

# the GPT of the reference configurations 1 to 4
GPTS = {
    "c64": dict(vocab_size=256, n_embd=64, n_head=4, n_layer=2, block_size=512),
    "c256": dict(vocab_size=512, n_embd=256, n_head=8, n_layer=4, block_size=2048),
    "c512": dict(vocab_size=1024, n_embd=512, n_head=8, n_layer=6, block_size=4096),
    "c768": dict(vocab_size=4096, n_embd=768, n_head=12, n_layer=12, block_size=2048),
}
# the design runs' sizes; Kipolix takes the second row's keys beside the first's
SIZES = {
    "w1024": dict(width=1024, heads=16, dim=64, kv_rank=256, ff=4096, window=512,
                  kv_heads=4, ret_dim=64, gated_ff=2736),
    "w2048": dict(width=2048, heads=16, dim=128, kv_rank=512, ff=8192, window=1024,
                  kv_heads=4, ret_dim=128, gated_ff=5456),
    "w2048_long": dict(width=2048, heads=16, dim=128, kv_rank=256, ff=8192, window=4096,
                       kv_heads=8, ret_dim=128, gated_ff=5456),
}
VOCAB, KEEP_FIRST, STREAMS, BUCKETS = 16384, 4, 4, 65521


def listed():
    return [
        # a hundred futures of one short series (reference configuration 1): one graph replay per token, all latency
        dict(name="predict_small", kind="predict", model="c64", rows=90, columns=1, horizon=48, samples=100, dtype="f32"),
        # the smallest calls: one request followed token by token
        dict(name="gpt_steps", kind="steps", family="gpt", model="c64", layers=2, requests=1, portion=24, singles=8, dtype="f32"),
        # batch scoring of short sequences (reference configuration 2, heads of 32)
        dict(name="gpt_forward", kind="forward", family="gpt", model="c256", layers=4, batch=256, tokens=512, dtype="bf16"),
        # the headline: 4096 futures of one series (reference configuration 4, with predict_samples' own sampler)
        dict(name="gpt_mc_decode", kind="decode", family="gpt", model="c768", layers=12, series=1, samples=4096, prompt=1024,
             horizon=256, free=True, top_p=1.0, dtype="bf16"),
        # a back-test: several series, ragged sizes, shared prompts, nucleus sampling of what is not given
        dict(name="gpt_backtest", kind="decode", family="gpt", model="c768", layers=12, series=3, samples=333, prompt=777,
             horizon=41, free=False, top_p=0.9, dtype="bf16"),
        # many long multivariate series, one trajectory each: prefill of long prompts, decoding against private caches
        # (reference configuration 3, a third of its horizon)
        dict(name="gpt_many_series", kind="decode", family="gpt", model="c512", layers=6, series=64, samples=1, prompt=3570,
             horizon=224, free=False, top_p=1.0, dtype="bf16"),
        # long-context attention (reference configuration 5)
        dict(name="attention_long", kind="attention", batch=8, heads=16, dim=128, tokens=8192),
        # one long prompt, all logits
        dict(name="delunex_forward", kind="forward", family="delunex", model="w2048", layers=8, batch=1, tokens=8192, dtype="bf16"),
        # batch serving: 256 rows behind prompts that four rows share
        dict(name="delunex_decode", kind="decode", family="delunex", model="w2048", layers=8, series=64, samples=4, prompt=1024,
             horizon=64, free=False, top_p=1.0, dtype="bf16"),
        # scoring a batch of medium sequences
        dict(name="kipolix_forward", kind="forward", family="kipolix", model="w1024", layers=8, batch=8, tokens=2048, dtype="bf16"),
        dict(name="kipolix_decode", kind="decode", family="kipolix", model="w2048", layers=8, series=256, samples=1, prompt=512,
             horizon=64, free=False, top_p=1.0, dtype="bf16"),
        # three requests fed a portion and then token by token, as a trace replay does
        dict(name="kipolix_steps", kind="steps", family="kipolix", model="w1024", layers=8, requests=3, portion=150, singles=12, dtype="bf16"),
    ]


def _log(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(("predict", "forward", "forward", "steps", "steps", "decode", "decode", "decode", "attention"))
    if kind == "predict":
        columns = rng.choice((1, 1, 2, 3))
        return dict(kind=kind, model="c64", rows=rng.randint(20, 90), columns=columns, horizon=_log(rng, 4, 48),
                    samples=_log(rng, 1, 400), dtype="f32")
    if kind == "attention":
        dim, tokens = rng.choice((32, 64, 128, 128)), _log(rng, 512, 16384)
        rows = max(1, 8 * 16 * 8192 // tokens)  # (sequence, head) pairs
        heads = rng.choice((8, 12, 16))
        return dict(kind=kind, batch=_log(rng, 1, max(1, min(32, rows // heads))), heads=heads, dim=dim, tokens=tokens)
    family = rng.choice(("gpt", "gpt", "delunex", "kipolix"))
    model = rng.choice(("c256", "c512", "c768") if family == "gpt" else ("w1024", "w2048", "w2048_long"))
    layers = rng.randint(2, GPTS[model]["n_layer"] if family == "gpt" else 8)
    base = dict(kind=kind, family=family, model=model, layers=layers, dtype="bf16")
    if kind == "forward":
        tokens = _log(rng, 16, 2048 if family == "gpt" else 8192)
        base["dtype"] = rng.choice(("bf16", "bf16", "bf16", "f32")) if model in ("c256", "c512") else "bf16"
        return dict(base, batch=_log(rng, 1, max(1, min(256, 32768 // tokens))), tokens=tokens)
    if kind == "steps":
        return dict(base, requests=rng.randint(1, 4), portion=_log(rng, 2, 700), singles=rng.randint(2, 16))
    samples = _log(rng, 1, 1200)
    prompt = _log(rng, 24, 1400 if family == "gpt" else 1500)
    series = _log(rng, 1, max(1, min(48, 1200 // samples, 60000 // prompt)))
    free = family == "gpt" and rng.random() < 0.4
    return dict(base, series=series, samples=samples, prompt=prompt, horizon=_log(rng, 8, 100), free=free,
                top_p=rng.choice((0.9, 1.0)) if family == "gpt" and not free else 1.0)


# ---- configurations and weights ------------------------------------------------------------
def gpt_config(case):
    c = dict(GPTS[case["model"]])
    if "layers" in case:
        c["n_layer"] = case["layers"]
    return c


def delunex_config(case):
    z, layers = SIZES[case["model"]], []
    for i in range(case["layers"]):
        m = dict(heads=z["heads"], dim=z["dim"], vdim=z["dim"], kv_rank=z["kv_rank"], scale=z["dim"] ** -0.5, mask={"size": z["window"]})
        if i % 2:
            m["kv_from"] = i - 1
        layers.append({"type": "latent_attention", "mixer": m, "mlp": {"kind": "dense", "ff": z["ff"]}})
    return {"architecture": "Delunex", "width": z["width"], "vocab": VOCAB, "canon": {"taps": 4}, "norm": {"eps": 1e-6},
            "embedding": {"scale": z["width"] ** 0.5}, "logit_scale": 1.0, "layers": layers}


def kipolix_config(case):
    z, layers = SIZES[case["model"]], []
    for i in range(case["layers"]):
        n, mlp = z["heads"], {"kind": "dense", "ff": z["gated_ff"]}
        if i % 4 == 0:
            m = dict(heads=n, dim=z["ret_dim"], vdim=z["ret_dim"], rot={"dims": z["ret_dim"], "base": 1e4},
                     decay=[1 - 2.0 ** (-5 - 6 * j / (n - 1)) for j in range(n)])
            layers.append({"type": "retention", "mixer": m, "mlp": mlp})
        else:
            m = dict(heads=n, kv_heads=z["kv_heads"], dim=z["dim"], vdim=z["dim"], scale=z["dim"] ** -0.5,
                     rot={"dims": z["dim"], "base": 1e4}, mask={"size": z["window"], "keep_first": KEEP_FIRST})
            layers.append({"type": "attention", "mixer": m, "mlp": mlp})
    return {"architecture": "Kipolix", "width": z["width"], "vocab": VOCAB, "streams": STREAMS, "norm": {"eps": 1e-6},
            "embedding": {"bigram": {"buckets": BUCKETS, "mul_prev": 8191, "mul_cur": 31}},
            "loop": {"start": 0, "stop": 0, "times": 1}, "layers": layers}


def config(case):
    return {"gpt": gpt_config, "delunex": delunex_config, "kipolix": kipolix_config}[case.get("family", "gpt")](case)


def weights(case, seed):
    """{checkpoint name: tensor on the GPU}.  GPT: all N(0, 0.02), as the reference configurations.  The others: linear
    layers that keep the scale of what they read, norm weights scattered around the value that leaves it alone."""
    dt, cfg, w = DTYPES[case["dtype"]], config(case), {}
    g = torch.Generator(device="cuda").manual_seed(7919 * seed + 1)

    def n(std, *s, mean=0.0):
        return (torch.randn(s, generator=g, device="cuda") * std + mean).to(dt)

    def lin(o, i):
        return n(0.8 / math.sqrt(i), o, i)

    if case.get("family", "gpt") == "gpt":
        C = cfg["n_embd"]
        w["token_embedding_table.weight"] = n(0.02, cfg["vocab_size"], C)
        for i in range(cfg["n_layer"]):
            p = f"blocks.{i}."
            for name in ("c_q", "c_k", "c_v", "c_g", "c_proj"):
                w[f"{p}sa.{name}.weight"] = n(0.02, C, C)
            w[p + "ffwd.net.0.weight"], w[p + "ffwd.net.2.weight"] = n(0.02, 4 * C, C), n(0.02, C, 2 * C)
            w[p + "attn_res_proj.weight"], w[p + "mlp_res_proj.weight"] = n(0.02, 1, C), n(0.02, 1, C)
        return w
    C, V = cfg["width"], cfg["vocab"]
    kip = case["family"] == "kipolix"
    w["embed"] = n(1.0 if kip else 1.0 / math.sqrt(C), V, C)
    w["final.norm"] = n(0.1, C, mean=0.0 if kip else 1.0)
    if kip:
        w["bigram"], w["head"] = n(0.7, BUCKETS + 1, C), lin(V, C)
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        H, d = m["heads"], m["dim"]
        w[p + "mix.q"], w[p + "mix.o"] = lin(H * d, C), lin(C, H * d)
        if kip:
            G = m.get("kv_heads", H)
            w[p + "mix.k"], w[p + "mix.v"] = lin(G * d, C), lin(G * d, C)
            if layer["type"] == "retention":
                w[p + "mix.g"] = lin(H * d, C)
            else:
                w[p + "mix.q.norm"], w[p + "mix.k.norm"] = n(0.1, H * d, mean=1.0), n(0.1, G * d, mean=1.0)
            w[p + "mlp.gate"] = lin(ff, C)
            for q in (1, 2):
                w[f"{p}norm{q}"] = n(0.1, C)
                w[f"{p}hc{q}.in"], w[f"{p}hc{q}.out"] = n(0.05, STREAMS, mean=1 / STREAMS), n(0.1, STREAMS, mean=0.4)
                w[f"{p}hc{q}.mix"] = (0.9 * torch.eye(STREAMS, device="cuda") + n(0.05, STREAMS, STREAMS).float()).to(dt)
        else:
            r = m["kv_rank"]
            if "kv_from" not in m:
                w[p + "mix.dkv"], w[p + "mix.dkv.norm"] = lin(r, C), n(0.1, r, mean=1.0)
            w[p + "mix.uk"], w[p + "mix.uv"], w[p + "mix.g"] = lin(H * d, r), lin(H * d, r), lin(H, C)
            w[p + "norm1"], w[p + "norm2"] = n(0.1, C, mean=0.7), n(0.1, C, mean=0.7)
            w[p + "mlp.act"], w[p + "canon1"] = n(0.1, 2, mean=0.3), n(0.2, C, 4)
            a = torch.randn(i + 2, generator=g, device="cuda") * 0.1
            a[-1] += 1.0
            w[p + "dwa"] = a.to(dt)
        w[p + "mlp.up"], w[p + "mlp.down"] = lin(ff, C), lin(C, ff)
    return w


def vocabulary(case):
    c = config(case)
    return c["vocab_size"] if case.get("family", "gpt") == "gpt" else c["vocab"]


def token_ids(case, seed, *shape):
    """Tokens of random-walk series for the GPT (a band around the middle of the vocabulary), of text otherwise."""
    V = vocabulary(case)
    g = torch.Generator(device="cuda").manual_seed(104729 * seed + 2)
    if case.get("family", "gpt") == "gpt":
        z = torch.randn(shape, generator=g, device="cuda") * (V / 10) + V / 2
        return z.round().clamp(0, V - 1).to(torch.int64)
    return torch.randint(0, V, shape, generator=g, device="cuda")


def series_frame(case, seed):
    """Random walks with a season, [rows, columns]."""
    rng = np.random.default_rng(seed + 11)
    t = np.arange(case["rows"])[:, None]
    walk = np.cumsum(rng.normal(0.0, 1.0, (case["rows"], case["columns"])), axis=0)
    return walk + np.sin(2 * np.pi * t / 24.0)


def attention_inputs(case, seed):
    B, H, D, T = case["batch"], case["heads"], case["dim"], case["tokens"]
    g = torch.Generator(device="cuda").manual_seed(31 * seed + 5)
    return torch.randn((B * T, 3 * H * D), generator=g, device="cuda").to(torch.bfloat16)


def rotation(D, positions, dtype, theta=10000.0):
    """[positions, D / 2, 2]: cos and sin as the reference's buffer holds them in the model's dtype."""
    f = 1.0 / (theta ** (torch.arange(0, D, 2, dtype=torch.float32) / D))
    ang = torch.outer(torch.arange(positions, dtype=torch.float32), f)
    return torch.stack([ang.cos(), ang.sin()], dim=-1).to(dtype).cuda()


# ---- what a user's program has, and one pass ------------------------------------------------
def build(case, seed):
    from diff_gpt_b200 import GPT, Delunex, Kipolix

    cls = {"gpt": GPT, "delunex": Delunex, "kipolix": Kipolix}[case.get("family", "gpt")]
    with torch.device("cuda"):
        m = cls.from_config(config(case))
    m = m.to(DTYPES[case["dtype"]]).cuda().eval()
    m.load_tensors(weights(case, seed))
    return m


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "attention":
        from diff_gpt_b200 import ops

        B, H, D, T = case["batch"], case["heads"], case["dim"], case["tokens"]
        cache = torch.empty((B, 2, H, T, D), device="cuda", dtype=torch.bfloat16)
        return dict(
            s, qkv=attention_inputs(case, seed), cache=cache, table=rotation(D, T, torch.bfloat16).contiguous(), dims=(B, H, D, T),
            layout=ops.kv_layout(cache[0, 0], cache[0, 1], 2 * H * T * D, T * D, T), zero=torch.zeros(B, dtype=torch.int32, device="cuda"),
            status=torch.zeros(1, dtype=torch.int32, device="cuda"),
        )
    model = build(case, seed)
    if kind == "predict":
        import pandas as pd

        from diff_gpt_b200 import TemperatureSampler
        from diff_gpt_b200.diff_gpt import DiffGPT
        from diff_gpt_b200.encoder_decoder import get_domain_of_definition

        x = series_frame(case, seed)
        dom = get_domain_of_definition(x, 1, use_decimal=False)
        dg = DiffGPT(model=model, order_of_derivative=1, domain_of_definition=dom, use_decimal=False)
        frame = pd.DataFrame(x, columns=[f"y{i}" for i in range(case["columns"])])
        return dict(s, dg=dg, frame=frame, horizon=case["horizon"], samples=case["samples"], sampler=TemperatureSampler(1.0))
    if kind == "forward":
        return dict(s, model=model, idx=token_ids(case, seed, case["batch"], case["tokens"]))
    if kind == "steps":
        from diff_gpt_b200 import StepRunner

        n = case["portion"] + case["singles"]
        return dict(s, runner=StepRunner(model), tokens=token_ids(case, seed, case["requests"], n).tolist(), portion=case["portion"])
    from diff_gpt_b200 import NucleusSampler, TemperatureSampler
    from diff_gpt_b200.model.engine import DecodeRun

    S, P, G = case["series"], case["prompt"], case["horizon"]
    ids = token_ids(case, seed, S, P + G)
    prompts = ids[:, :P].to(torch.int32).contiguous()
    force = None if case["free"] else [row[:-1] + [None] for row in ids[:, P:].tolist()]
    sampler = NucleusSampler(case["top_p"], TemperatureSampler(1.0)) if case["top_p"] < 1.0 else TemperatureSampler(1.0)
    with torch.inference_mode():
        run_ = DecodeRun(model, prompts, case["samples"], G, sampler, 42, force, fused_head=case["free"])
    return dict(s, run=run_, prompts=prompts, force=force, free=case["free"])


@torch.inference_mode()
def run(s):
    kind = s["kind"]
    if kind == "predict":
        return s["dg"].predict_samples(s["frame"], s["horizon"], s["samples"], sampler=s["sampler"])
    if kind == "forward":
        return s["model"](s["idx"])[0]
    if kind == "steps":
        runner, portion, out = s["runner"], s["portion"], []
        for r, tokens in enumerate(s["tokens"]):
            out.append(runner.step(r, tokens[:portion], [portion - 1]))
        for t in range(portion, len(s["tokens"][0])):
            for r, tokens in enumerate(s["tokens"]):
                out.append(runner.step(r, tokens[t : t + 1], [0]))
        for r in range(len(s["tokens"])):
            runner.finish(r)
        return torch.cat(out)
    if kind == "decode":
        r = s["run"]
        r.load(s["prompts"], s["force"])
        r.start()
        r.advance(r.G)
        r.check_status()
        return {"prompt_logits": r.logits0, "tokens": r.tokens_so_far()} if s["free"] else {"logits": r.logits, "tokens": r.tokens_so_far()}
    from diff_gpt_b200 import ops

    B, H, D, T = s["dims"]
    C, qkv = H * D, s["qkv"]
    q = torch.empty((B * T, C), device="cuda", dtype=torch.bfloat16)
    y = torch.empty_like(q)
    ops.rope_qknorm_kvappend(qkv[:, :C], qkv[:, C : 2 * C], qkv[:, 2 * C :], q, s["table"], s["layout"], s["zero"], s["zero"], None, B, T, H, D,
                             s["status"])
    ops.fmha_prefill(q, s["layout"], y, B=B, H=H, Tq=T, D=D, q_batch_stride=T * C, q_row_stride=C, o_batch_stride=T * C, o_row_stride=C,
                     kv_len_all=T, causal=True, status=s["status"])
    return {"q": q, "y": y, "cache": s["cache"]}


# ---- what a pass cannot do without --------------------------------------------------------------
def _model_work(case):
    """(multiply-adds of one token's products without the head, those of the head, bytes of the weights that a pass reads whole)"""
    cfg = config(case)
    if case.get("family", "gpt") == "gpt":
        C = cfg["n_embd"]
        per, head = cfg["n_layer"] * 11 * C * C, cfg["vocab_size"] * C
    else:
        C, per = cfg["width"], 0
        for layer in cfg["layers"]:
            m, ff = layer["mixer"], layer["mlp"]["ff"]
            H, d = m["heads"], m["dim"]
            if case["family"] == "delunex":
                per += 2 * C * H * d + C * H + 2 * C * ff + (C * m["kv_rank"] if "kv_from" not in m else 0) + 2 * H * d * m["kv_rank"]
            elif layer["type"] == "retention":
                per += 5 * C * H * d + 3 * C * ff
            else:
                per += 2 * C * H * d + 2 * C * m["kv_heads"] * d + 3 * C * ff
        head = cfg["vocab"] * C
    size = 4 if case["dtype"] == "f32" else 2
    return per, head, size * (per + head)


def _mixers(case):
    """For every layer (multiply-adds per query and key, bytes of one cached key, the most keys a query sees); a retention
    layer has a state instead: no keys, `state` bytes."""
    cfg, size = config(case), 4 if case["dtype"] == "f32" else 2
    if case.get("family", "gpt") == "gpt":
        C = cfg["n_embd"]
        return [(2 * C, 2 * C * size, 1 << 40, 0)] * cfg["n_layer"]
    out = []
    for layer in cfg["layers"]:
        m = layer["mixer"]
        H, d = m["heads"], m["dim"]
        if case["family"] == "delunex":
            out.append((2 * H * d, m["kv_rank"] * size, m["mask"]["size"], 0))
        elif layer["type"] == "retention":
            out.append((0, 0, 0, H * d * d * 4))
        else:
            out.append((2 * H * d, 2 * m["kv_heads"] * d * size, m["mask"]["size"] + KEEP_FIRST, 0))
    return out


def _seen(first, last, most):
    """Sum over queries first .. last - 1 of the keys they see (query i sees i + 1, at most `most`)."""
    grow = min(max(most, first), last)
    return (grow * (grow + 1) - first * (first + 1)) // 2 + (last - grow) * most


def _sequence(case, T, logits):
    """(bytes, flops) of a whole sequence without the weights' bytes."""
    per, head, _ = _model_work(case)
    flops = 2 * (per * T + head * logits)
    for macs, _key, most, state in _mixers(case):
        flops += 2 * macs * _seen(0, T, most) + (4 * state // 4 * T if state else 0)
    return 4 * T + logits * vocabulary(case) * (4 if case["dtype"] == "f32" else 2), flops


def work(case):
    kind = case["kind"]
    if kind == "attention":
        B, H, D, T = case["batch"], case["heads"], case["dim"], case["tokens"]
        return {"bytes": 2 * B * T * H * D * (3 + 4), "flops": 2 * B * H * D * T * (T + 1)}
    per, head, size = _model_work(case)
    if kind == "forward":
        b, f = _sequence(case, case["tokens"], case["tokens"])
        return {"bytes": size + case["batch"] * b, "flops": case["batch"] * f}
    if kind == "steps":
        S, N, P, G = case["requests"], 1, case["portion"], case["singles"] + 1
    elif kind == "predict":
        S, N, P, G = 1, case["samples"], (case["rows"] - 1) * case["columns"], case["horizon"] * case["columns"]
    else:
        S, N, P, G = case["series"], case["samples"], case["prompt"], case["horizon"]
    # the prompts, then G - 1 steps that each read the weights, the shared keys of every series and each row's own
    b, f = _sequence(case, P, 1)
    total, flops, R = size + S * b, S * f, S * N
    steps = G - 1 if kind != "steps" else S * (G - 1)  # given tokens come one request at a time
    total += steps * size
    flops += 2 * R * (G - 1) * (per + head)
    for macs, key, most, state in _mixers(case):
        flops += 2 * R * macs * _seen(P, P + G - 1, most)
        own = _seen(0, G - 1, most)
        total += key * (R * own + S * (_seen(P, P + G - 1, most) - own)) + 2 * state * R * (G - 1)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """About four times what was measured: the error against `exact` (bf16 logits 4e-3 to 8e-3, attention 2e-3 to 3.5e-3, fp32
    logits 2e-7 to 2e-6); and, for drawn tokens, what two orders of the same bf16 sums (prompt keys read by the shared phase
    or by the per-row kernel) change: 0.5 % of 256 x 1024 free draws, 15 % of the one nucleus draw behind forced tokens,
    none of 400 x 48 fp32 draws (there, one future in a hundred taking another path is 0.02 or less)."""
    f32 = case.get("dtype", "bf16") == "f32"
    if case["kind"] == "attention":
        return {"rel": 0.012}
    if case["kind"] == "predict":
        return {"rel": 0.02}
    rel = 1e-5 if f32 else 0.03
    if case["kind"] != "decode":
        return {"rel": rel}
    G, R = case["horizon"], case["series"] * case["samples"]
    return {"rel": rel, "differ": min(0.5, 0.02 + 8 / (R * G) if case["free"] else 0.6 / G + 1 / (R * G))}


# ---- the same in 64 bits ---------------------------------------------------------------------------
def _norm(x, eps=torch.finfo(torch.float32).eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window=None, keep=0):
    """q [T, H, d], k and v [T, G, d] in float64, causal, with a window and kept first keys; a block of queries at a time."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out, step = torch.empty_like(q), max(256, (1 << 27) // (T * 8))
    j = torch.arange(T, device=q.device)
    for a in range(0, T, step):
        b = min(T, a + step)
        i = j[a:b, None]
        seen = j[None, :b] <= i
        if window is not None:
            seen &= (i - j[None, :b] < window) | (j[None, :b] < keep)
        for h in range(H):
            p = ((q[a:b, h] @ k[:b, h * G // H].T) * scale).masked_fill_(~seen, -math.inf)
            out[a:b, h] = torch.softmax(p, -1) @ v[:b, h * G // H]
    return out


def _pairs(x, c, s):
    """x [T, H, d]: dimension 2 i turned with 2 i + 1."""
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)


def _gpt64(cfg, w, ids, last, dt):
    C, H = cfg["n_embd"], cfg["n_head"]
    T, D = ids.shape[0], C // H
    cs = rotation(D, T, dt).double()[:, None]
    c, s = cs[..., 0], cs[..., 1]
    x = _norm(w["token_embedding_table.weight"][ids])
    done, part = [x], x

    def mix(name):
        v = torch.stack(done + [part])
        a = torch.softmax(_norm(v) @ w[name].reshape(-1), 0)
        return _norm((a[..., None] * v).sum(0))

    for i in range(cfg["n_layer"]):
        p = f"blocks.{i}."
        u = mix(p + "attn_res_proj.weight") if i else _norm(x)
        done, part = done + [part], None
        q, k, v, g = (u @ w[f"{p}sa.c_{n}.weight"].T for n in "qkvg")
        q, k = (_norm(_pairs(t.view(T, H, D), c, s)) for t in (q, k))
        y = _attend(q, k, v.view(T, H, D), D**-0.5).reshape(T, C) * torch.sigmoid(g)
        part = y @ w[p + "sa.c_proj.weight"].T
        f = mix(p + "mlp_res_proj.weight") @ w[p + "ffwd.net.0.weight"].T
        gate, lin = f[..., 0::2].clamp(max=7.0), f[..., 1::2].clamp(-7.0, 7.0)
        part = part + (gate * torch.sigmoid(1.702 * gate) * (lin + 1)) @ w[p + "ffwd.net.2.weight"].T
    return _norm(part[-1:] if last else part) @ w["token_embedding_table.weight"].T


def _delunex64(cfg, w, ids, last, dt):
    eps, T = cfg["norm"]["eps"], ids.shape[0]
    x = w["embed"][ids] * cfg["embedding"]["scale"]
    states, lat = [x], {}
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        H, d = m["heads"], m["dim"]
        taps = w[p + "canon1"]
        h = x + sum(taps[:, j] * F.pad(x, (0, 0, 3 - j, 0))[:T] for j in range(4))
        if "kv_from" not in m:
            lat[i] = _norm(h @ w[p + "mix.dkv"].T, eps) * w[p + "mix.dkv.norm"]
        c = lat[m.get("kv_from", i)]
        q, k, v = ((t @ w[p + n].T).view(T, H, d) for t, n in ((h, "mix.q"), (c, "mix.uk"), (c, "mix.uv")))
        y = _attend(q, k, v, m["scale"], m["mask"]["size"]) * torch.sigmoid(h @ w[p + "mix.g"].T)[..., None]
        x = x + _norm(y.reshape(T, -1) @ w[p + "mix.o"].T, eps) * w[p + "norm1"]
        z = x @ w[p + "mlp.up"].T
        ap, an = F.softplus(w[p + "mlp.act"][0]), 0.5 + F.softplus(w[p + "mlp.act"][1])
        low = z.clamp(max=0.0)
        z = torch.where(z > 0, ap * z * z, an * (torch.expm1(low) - low)) + z / 2
        x = x + _norm(z @ w[p + "mlp.down"].T, eps) * w[p + "norm2"]
        states.append(x)
        x = sum(a * t for a, t in zip(w[p + "dwa"], states))
    return _norm(x[-1:] if last else x, eps) * w["final.norm"] @ w["embed"].T


def _kipolix64(cfg, w, ids, last, dt):
    eps, T, big = cfg["norm"]["eps"], ids.shape[0], cfg["embedding"]["bigram"]
    rows = torch.full_like(ids, BUCKETS)
    rows[1:] = (ids[:-1] * big["mul_prev"] + ids[1:] * big["mul_cur"]) % BUCKETS
    x = (w["embed"][ids] + w["bigram"][rows]).expand(STREAMS, -1, -1)
    t = torch.arange(T, dtype=torch.float64, device=ids.device)

    def retention(h, m, p):
        H, d = m["heads"], m["dim"]
        q, k, v = ((h @ w[p + n].T).view(T, H, d) for n in ("mix.q", "mix.k", "mix.v"))
        a = t[:, None] * m["rot"]["base"] ** (-2.0 * torch.arange(d // 2, dtype=torch.float64, device=t.device) / d)
        c, s = a.cos()[:, None], a.sin()[:, None]
        q, k = (torch.cat([z[..., : d // 2] * c - z[..., d // 2 :] * s, z[..., d // 2 :] * c + z[..., : d // 2] * s], -1) for z in (q, k))
        o, step = torch.empty_like(q), max(256, (1 << 27) // (T * 8))
        for n in range(H):
            for lo in range(0, T, step):
                hi = min(T, lo + step)
                gap = t[lo:hi, None] - t[None, :hi]
                fade = torch.where(gap >= 0, m["decay"][n] ** gap.clamp(min=0), 0.0)
                o[lo:hi, n] = ((q[lo:hi, n] @ k[:hi, n].T) * d**-0.5 * fade) @ v[:hi, n]
        return _norm(o, eps).reshape(T, -1) * F.silu(h @ w[p + "mix.g"].T)

    def attention(h, m, p):
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        q = (_norm(h @ w[p + "mix.q"].T, eps) * w[p + "mix.q.norm"]).view(T, H, d)
        k = (_norm(h @ w[p + "mix.k"].T, eps) * w[p + "mix.k.norm"]).view(T, G, d)
        a = t[:, None] * m["rot"]["base"] ** (-2.0 * torch.arange(d // 2, dtype=torch.float64, device=t.device) / d)
        c, s = a.cos()[:, None], a.sin()[:, None]
        y = _attend(_pairs(q, c, s), _pairs(k, c, s), (h @ w[p + "mix.v"].T).view(T, G, d), m["scale"], m["mask"]["size"], KEEP_FIRST)
        return y.reshape(T, -1)

    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        for q in (1, 2):
            h = torch.einsum("s,stc->tc", w[f"{p}hc{q}.in"], x)
            h = _norm(h, eps) * (1 + w[f"{p}norm{q}"])
            if q == 1:
                y = (retention if layer["type"] == "retention" else attention)(h, m, p) @ w[p + "mix.o"].T
            else:
                y = (F.silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
            x = torch.einsum("su,stc->utc", w[f"{p}hc{q}.mix"], x) + w[f"{p}hc{q}.out"][:, None, None] * y
    x = x.sum(0)
    return _norm(x[-1:] if last else x, eps) * (1 + w["final.norm"]) @ w["head"].T


def _logits64(case, w, ids, last):
    cfg = config(case)
    f = {"gpt": _gpt64, "delunex": _delunex64, "kipolix": _kipolix64}[case["family"]]
    return f(cfg, w, ids, last, DTYPES[case["dtype"]])


@torch.inference_mode()
def exact(case, seed):
    kind = case["kind"]
    if kind == "predict":
        return None  # drawn
    if kind == "attention":
        B, H, D, T = case["batch"], case["heads"], case["dim"], case["tokens"]
        qkv = attention_inputs(case, seed).view(B, T, 3, H, D)
        cs = rotation(D, T, torch.bfloat16).double()[:, None]
        q, y = (torch.empty((B, T, H, D), dtype=torch.float32, device="cuda") for _ in range(2))
        cache = torch.empty((B, 2, H, T, D), dtype=torch.float32, device="cuda")
        for b in range(B):
            qb, kb, vb = qkv[b].double().unbind(1)
            qb, kb = (_norm(_pairs(z, cs[..., 0], cs[..., 1])) for z in (qb, kb))
            q[b], y[b] = qb, _attend(qb, kb, vb, D**-0.5)
            cache[b, 0], cache[b, 1] = kb.transpose(0, 1), vb.transpose(0, 1)
        return {"q": q.view(B * T, -1), "y": y.view(B * T, -1), "cache": cache}
    w = {k: v.double() for k, v in weights(case, seed).items()}

    def capped(z):
        return 15.0 * torch.tanh(z / 15.0) if case["family"] == "gpt" else z

    if kind == "forward":
        idx = token_ids(case, seed, case["batch"], case["tokens"])
        return torch.stack([capped(_logits64(case, w, row, False)).float() for row in idx])
    if kind == "steps":
        P = case["portion"]
        ids = token_ids(case, seed, case["requests"], P + case["singles"])
        z = torch.stack([capped(_logits64(case, w, row, False))[P - 1 :] for row in ids])  # [requests, singles + 1, V]
        return torch.cat([z[:, 0], z[:, 1:].transpose(0, 1).flatten(0, 1)])
    S, P, G = case["series"], case["prompt"], case["horizon"]
    ids = token_ids(case, seed, S, P + G)
    if case["free"]:
        z = torch.cat([_logits64(case, w, row[:P], True) for row in ids])
        return {"prompt_logits": z, "tokens": None}
    z = torch.cat([_logits64(case, w, row[: P + G - 1], True) for row in ids])
    return {"logits": z.repeat_interleave(case["samples"], 0), "tokens": None}
