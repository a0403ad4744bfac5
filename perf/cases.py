"""The work that is timed: decode steps and prompts of the three decoder families, through their drivers, at the sizes
that ``bench.py`` and the tests use and over the ranges around them.

A case is a dict of plain values.  ``kind`` is the family: ``dsa`` (FP8 weights, latent attention over selected keys),
``dsa_mtp`` (the same with the prediction layer: prompts in chunks of four rows), ``ralasun`` (grouped-query attention,
routed experts), ``rozesun`` (attention over a latent cache, dense feed-forwards).  ``tokens`` 1 is a decode step at
position ``ctx``, more is a prompt behind ``ctx`` positions that the caches hold already."""

from __future__ import annotations

import math

import torch

import tilert_b200
from tilert_b200 import synthetic

F64, BF16, F32 = torch.float64, torch.bfloat16, torch.float32
VOCAB = 32768
PORTION = 2048   # most tokens of a prompt that the drivers run at once
DSA_VOCAB = 16160  # one of eight slices of 129280

RALASUN = {  # width: heads, kv_heads, experts, top, ff, shared_ff, window
    2048: (16, 4, 64, 6, 1408, 2816, 1024), 4096: (32, 8, 64, 8, 1536, 1536, 2048), 7168: (64, 8, 48, 8, 2048, 2048, 4096)}
ROZESUN = {  # width: heads, q_rank, kv_rank, ff, window
    2048: (16, 768, 512, 5632, 1024), 4096: (32, 1536, 512, 11264, 1024), 7168: (64, 1536, 512, 18432, 1024)}


def _ralasun(width: int, tokens: int, ctx: int, layers: int, sampled: bool = False) -> dict:
    heads, kv, experts, top, ff, sff, window = RALASUN[width]
    return {"kind": "ralasun", "width": width, "heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "experts": experts, "top": top,
            "ff": ff, "shared_ff": sff, "window": window, "layers": layers, "ctx": ctx, "tokens": tokens, "dtype": "bfloat16",
            "sampled": sampled}


def _rozesun(width: int, tokens: int, ctx: int, layers: int, sampled: bool = False) -> dict:
    heads, q_rank, kv_rank, ff, window = ROZESUN[width]
    return {"kind": "rozesun", "width": width, "heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": q_rank, "kv_rank": kv_rank,
            "ff": ff, "window": window, "layers": layers, "ctx": ctx, "tokens": tokens, "dtype": "bfloat16", "sampled": sampled}


def listed() -> list[dict]:
    exact_mode = {"kind": "ralasun", "width": 1024, "heads": 8, "kv_heads": 2, "dim": 96, "vdim": 64, "experts": 16, "top": 4, "ff": 704,
                  "shared_ff": 360, "window": 200, "layers": 2, "ctx": 0, "tokens": 97, "dtype": "float32", "sampled": False}
    return [
        # the workload of the benchmark: one token through FP8 layers at full width, a dense one and an expert one, with
        # a rank's slice of the head, 4K positions cached
        {"name": "dsa_token_4k", "kind": "dsa", "ctx": 4000, "rows": 4096, "experts": 256, "tokens": 1},
        # the same at a long context, where the indexer scans 128K keys
        {"name": "dsa_token_128k", "kind": "dsa", "ctx": 131000, "rows": 131072, "experts": 64, "tokens": 1},
        # a short prompt of the speculative runtime, four rows at a time, the last chunk ragged
        {"name": "dsa_prompt_mtp", "kind": "dsa_mtp", "ctx": 0, "rows": 4096, "experts": 64, "tokens": 30},
        # the smallest call: one token of a small model, where launches and latency count
        {"name": "ralasun_token_2048", **_ralasun(2048, 1, 1500, 3)},
        # one token of a large model: the weight stream
        {"name": "ralasun_token_7168", **_ralasun(7168, 1, 4500, 2)},
        # a full portion of a long prompt, every query with a full window behind it
        {"name": "ralasun_prompt_4096", **_ralasun(4096, 2048, 2048, 2)},
        # a user's first question: a ragged prompt on empty caches
        {"name": "ralasun_prompt_short", **_ralasun(2048, 173, 0, 3)},
        # one sampled token over latent caches, all keys in one layer and a window in the other
        {"name": "rozesun_token_4096", **_rozesun(4096, 1, 6000, 4, sampled=True)},
        # a full portion of a long prompt behind 4096 positions
        {"name": "rozesun_prompt_4096", **_rozesun(4096, 2048, 4096, 2)},
        # a follow-up question: few tokens on many cached positions
        {"name": "rozesun_prompt_short", **_rozesun(2048, 37, 4000, 4)},
        # the widest model, a document of odd length from the start
        {"name": "rozesun_prompt_7168", **_rozesun(7168, 1357, 0, 2)},
        # the exact 32-bit mode at small uneven sizes
        {"name": "ralasun_exact_mode", **exact_mode},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["dsa", "dsa_mtp", "ralasun", "ralasun", "ralasun", "rozesun", "rozesun", "rozesun"])
    if kind == "dsa":
        ctx = _log(rng, 40, 130000)
        return {"kind": kind, "ctx": ctx, "rows": (ctx // 256 + 1) * 256, "experts": 64, "tokens": 1}
    if kind == "dsa_mtp":
        return {"kind": kind, "ctx": 0, "rows": 2048, "experts": 64, "tokens": rng.randint(5, 40)}
    tokens = 1 if rng.random() < 0.3 else _log(rng, 2, 2048)
    ctx = rng.choice([0, _log(rng, 1, 4096), rng.randint(1, 4096)])
    if tokens == 1:
        ctx += 1
    width = rng.randint(120, 512) * 8 + rng.choice([0, 0, 2])
    dtype = "float32" if tokens <= 64 and width <= 1600 else "bfloat16"
    common = {"kind": kind, "width": width, "layers": 2, "ctx": ctx, "tokens": tokens, "dtype": dtype, "sampled": rng.random() < 0.25}
    if kind == "ralasun":
        kv = rng.choice([1, 2, 4, 8])
        group = rng.choice([1, 2, 3, 4, 6, 8])
        experts = rng.randint(4, 64)
        return common | {"heads": min(kv * group, 32 // kv * kv), "kv_heads": kv, "dim": rng.choice([64, 80, 96, 128]), "vdim": rng.choice([64, 72, 128]),
                         "experts": experts, "top": rng.randint(1, min(8, experts)), "ff": rng.randint(200, 1536),
                         "shared_ff": rng.choice([0, rng.randint(200, 2816)]), "window": rng.choice([0, rng.randint(30, 4096)])}
    return common | {"heads": rng.randint(4, 32), "dim": rng.choice([64, 96, 128]), "rot_dim": rng.choice([32, 64]), "vdim": rng.choice([64, 96, 128]),
                     "q_rank": rng.randint(300, 1536), "kv_rank": rng.choice([256, 384, 512]), "ff": rng.randint(1000, 11264),
                     "window": rng.randint(30, 2048)}


# ---------------------------------------------------------------- models and inputs
def _max_len(case: dict) -> int:
    return max(2048, case["ctx"] + case["tokens"] + 64)


def _args(case: dict):
    if case["kind"].startswith("dsa"):
        from dataclasses import replace

        from tilert_b200.models.deepseek_v3_2.model_args import ModelArgs

        return replace(ModelArgs(), n_layers=2, n_dense_layers=1, vocab_size=DSA_VOCAB, n_routed_experts=case["experts"])
    if case["kind"] == "ralasun":
        from tilert_b200.models.ralasun.model_args import MixerArgs, MlpArgs, uniform_args

        mix = MixerArgs(case["heads"], case["kv_heads"], case["dim"], case["vdim"], case["window"] or None, case["dim"] ** -0.5, True)
        mlp = MlpArgs(case["experts"], case["top"], case["ff"], 7.0, case["shared_ff"], 7.0)
        return uniform_args(case["layers"], case["width"], VOCAB, mix, mlp, max_seq_len=_max_len(case))
    from tilert_b200.models.rozesun.model_args import LayerArgs, MixerArgs, MlpArgs, RozesunArgs

    sizes = dict(heads=case["heads"], dim=case["dim"], rot_dim=case["rot_dim"], vdim=case["vdim"], q_rank=case["q_rank"], kv_rank=case["kv_rank"],
                 scale=(case["dim"] + case["rot_dim"]) ** -0.5, rot_base=1e4)
    kinds = (MixerArgs("latent_attention", **sizes), MixerArgs("latent_attention_2", window=case["window"], **sizes))
    return RozesunArgs(VOCAB, case["width"], 1e-6, 1.0, tuple(LayerArgs(kinds[i % 2], MlpArgs(case["ff"], 7.0)) for i in range(case["layers"])),
                       max_seq_len=_max_len(case))


def _weights(case: dict, seed: int) -> dict:
    args = _args(case)
    if case["kind"].startswith("dsa"):
        # Embeddings of unit size under layers that add less to them, as in a trained model: a key or an expert that two
        # correct implementations choose differently, because of a near tie, then changes a result by per cents at most.
        sd = synthetic.random_model_state_dict(args, "cuda", seed=seed, std=0.01, with_mtp=case["kind"] == "dsa_mtp")
        sd["model.embed_tokens.weight"] = sd["model.embed_tokens.weight"] * 100
        return sd
    make = synthetic.random_ralasun_state_dict if case["kind"] == "ralasun" else synthetic.random_rozesun_state_dict
    return make(args, "cuda", seed=seed)


def _tokens(case: dict, seed: int) -> list[int]:
    """The cached positions' tokens, then the pass's."""
    vocab = DSA_VOCAB if case["kind"].startswith("dsa") else VOCAB
    n = case["tokens"] + (0 if case["kind"] == "dsa" else case["ctx"])
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed * 31 + 7)).tolist()


def _dsa_caches(case: dict, seed: int) -> list[tuple[torch.Tensor, ...]]:
    """(ki, kv, pe) of the cached positions per layer, as an external prefill hands them over."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 17 + 3)
    return [tuple(torch.randn(case["ctx"], d, generator=gen, device="cuda").to(BF16) for d in (128, 512, 64)) for _ in range(2)]


def prepare(case: dict, seed: int) -> dict:
    torch.cuda.set_device(0)
    args, sd, toks = _args(case), _weights(case, seed), _tokens(case, seed)
    if case["kind"] == "dsa":
        from tilert_b200.models.deepseek_v3_2.model import DsaModel

        tilert_b200.load_backend("deepseek_v3_2")
        model = DsaModel(args, sd, cache_len=case["rows"])
        model.inject_cache(_dsa_caches(case, seed))
        state = {"model": model, "ctx": case["ctx"], "kind": "dsa", "token": toks[0]}
    elif case["kind"] == "dsa_mtp":
        from tilert_b200.models.deepseek_v3_2.mtp import MtpDsaModel

        tilert_b200.load_backend("deepseek_v3_2")
        state = {"model": MtpDsaModel(args, sd, cache_len=case["rows"]), "kind": "dsa_mtp", "prompt": toks}
    else:
        if case["kind"] == "ralasun":
            from tilert_b200.models.ralasun.model import RalasunModel as Model
        else:
            from tilert_b200.models.rozesun.model import RozesunModel as Model
        tilert_b200.load_backend("ralasun")
        model = Model(args, sd, dtype=case["dtype"])
        if case["sampled"]:
            model.set_sampling(temperature=0.8, top_p=0.95, top_k=50, use_top_p=True, seed=1234)
        state = {"model": model, "ctx": case["ctx"], "kind": "rows", "prompt": toks[case["ctx"]:], "sampled": case["sampled"]}
        if case["ctx"]:
            model.prefill(toks[: case["ctx"]])
    del sd
    torch.cuda.empty_cache()
    run(state)  # a serving program has taken its step's launches into a graph before
    torch.cuda.synchronize()
    return state


def run(state: dict) -> dict:
    model = state["model"]
    if state["kind"] == "dsa_mtp":
        # the prompt in chunks of four rows, as the generation loop feeds them
        prompt, n = state["prompt"], len(state["prompt"])
        model.reset_sequence()
        while model.pos < n:
            chunk = prompt[model.pos: model.pos + 4]
            valid = len(chunk)
            model.set_prefill_mtp_extra_token(prompt[model.pos + 4] if model.pos + 4 < n else prompt[-1])
            model.set_prefill_valid_tokens(valid)
            model.forward(chunk + [chunk[-1]] * (4 - valid))
        layers = [*model.layers, model.mtp_layer]
        last = (n - 1) % 4  # row of the last token in its chunk
        return {"logits": model.logits[0, : last + 1], "next": model.mtp_logits[0, : last + 1],
                "caches": [c[0, :n] for layer in layers for c in (layer.ki_cache, layer.kv_cache, layer.pe_cache)]}
    model.set_cur_pos(state["ctx"])
    if state["kind"] == "dsa":
        model.forward(state["token"], state["ctx"])
        return {"logits": model.logits, "caches": [c[0] for layer in model.layers for c in (layer.ki_cache, layer.kv_cache, layer.pe_cache)]}
    if len(state["prompt"]) == 1:
        model.forward(state["prompt"][0], state["ctx"])
        logits = model.logits.view(1, -1)
    else:
        logits = model.prefill(state["prompt"])
    out = {"logits": logits, "caches": [t for layer in model.layers for c in (getattr(layer, "caches", None) or [layer.cache]) for t in c._tensors()]}
    if state["sampled"]:
        out["top_logprobs"] = model.topn_logprobs
    return out


# ---------------------------------------------------------------- work
def _visible(case: dict, window: int) -> float:
    """Keys that the pass's queries see together, summed over them."""
    n, ctx = case["tokens"], case["ctx"]
    return float(sum(min(ctx + i + 1, window or ctx + i + 1) for i in range(n)))


def work(case: dict) -> dict:
    n, ctx = case["tokens"], case["ctx"]
    if case["kind"].startswith("dsa"):
        a = _args(case)
        d, h = a.dim, a.n_heads
        attn = d * (a.q_lora_rank + 512 + 64 + 128) + a.q_lora_rank * (h * 192 + 64 * 128) + h * 512 * 256 + d * h * 128
        expert = 3 * d * a.moe_inter_dim
        mtp = case["kind"] == "dsa_mtp"
        moe = 2 if mtp else 1
        chunks = [min(4, n - i) for i in range(0, n, 4)] if mtp else [1]
        used = sum(1 + a.n_routed_experts * (1 - (1 - 8 / a.n_routed_experts) ** c) for c in chunks)  # experts that are read, per expert layer
        fixed = (moe + 1) * attn + 3 * d * a.inter_dim
        plain = moe * 2 * d * a.n_routed_experts + (moe + 1) * 2 * d * 64 + moe * 2 * d * DSA_VOCAB + (4 * d * d if mtp else 0)  # bf16 weights
        keys = sum(range(1, n + 1)) if mtp else ctx + 1
        seen = keys if mtp else min(ctx + 1, a.index_topk)
        nbytes = len(chunks) * (fixed + plain) + moe * used * expert + (moe + 1) * (256 * (len(chunks) * n / 2 if mtp else keys) + 1152 * seen)
        flops = 2 * n * (fixed + plain / 2 + moe * 9 * expert) + (moe + 1) * 2 * (keys * 64 * 128 + seen * h * (512 + 576))
        return {"bytes": nbytes, "flops": flops}
    w, size, nl = case["width"], 4 if case["dtype"] == "float32" else 2, case["layers"]
    if case["kind"] == "ralasun":
        q, kv = case["heads"] * case["dim"], case["kv_heads"] * (case["dim"] + case["vdim"])
        attn_w = w * (q + kv + case["heads"] * case["vdim"])
        expert, shared = 3 * w * case["ff"], 3 * w * case["shared_ff"]
        used = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** n)
        weights = attn_w + w * case["experts"] + used * expert + shared
        per_token = attn_w + w * case["experts"] + case["top"] * expert + shared
        pairs = _visible(case, case["window"])
        cached = min(ctx, case["window"] + n - 1) if case["window"] else ctx
        nbytes = nl * (2 * weights + size * kv * (cached + n)) + 2 * w * VOCAB + 4 * VOCAB
        flops = 2 * nl * (n * per_token + pairs * case["heads"] * (case["dim"] + case["vdim"])) + 2 * w * VOCAB
        return {"bytes": nbytes, "flops": flops}
    nbytes, flops = 2 * w * VOCAB + 4 * VOCAB, 2 * w * VOCAB
    h, r, qk, v = case["heads"], case["kv_rank"], case["dim"] + case["rot_dim"], case["vdim"]
    for i in range(nl):
        window = case["window"] if i % 2 else 0
        gate = h if i % 2 else h * v
        weights = w * (case["q_rank"] + r + case["rot_dim"] + gate) + case["q_rank"] * h * qk + r * h * (case["dim"] + v) + w * h * v + 3 * w * case["ff"]
        cached = min(ctx, window + n - 1) if window else ctx
        pairs = _visible(case, window)
        expanded = pairs * h * (qk + v) + (cached + n) * r * h * (case["dim"] + v)
        absorbed = pairs * h * (2 * r + case["rot_dim"]) + n * r * h * (case["dim"] + v)
        nbytes += 2 * weights + size * (r + case["rot_dim"]) * (cached + n)
        flops += 2 * (n * (weights - r * h * (case["dim"] + v)) + min(expanded, absorbed))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case: dict) -> dict:
    """About four times the largest distance from ``exact`` over seeds and drawn cases.  bf16 activations alone give 0.5 %;
    the rest of ``dsa`` and ``ralasun`` is keys and experts chosen the other way at near ties."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    return {"rel": {"dsa": 0.1, "dsa_mtp": 0.1, "ralasun": 0.1, "rozesun": 0.02}[case["kind"]]}


# ---------------------------------------------------------------- plain 64-bit restatement
def _rms(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, b, eps=1e-6):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w.to(F64) + b.to(F64)


def _lin(x, w):
    return x @ w.to(F64).T


def _unit(x, gate, up, down, limit=7.0):
    g, u = _lin(x, gate).clamp(max=limit), _lin(x, up).clamp(-limit, limit)
    return _lin(g * torch.sigmoid(1.702 * g) * (u + 1), down)


def _attend(q, k, v, scale, window, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv]; one head and 1024 queries at a time."""
    t, h = q.shape[:2]
    out = torch.empty(t, h, v.shape[-1], dtype=F64, device=q.device)
    per = h // k.shape[1]
    pos = torch.arange(t, device=q.device)
    for lo in range(0, t, 1024):
        hi = min(lo + 1024, t)
        first = max(0, lo - window + 1) if window else 0
        gap = pos[lo:hi, None] - pos[None, first:hi]
        hidden = (gap < 0) | (gap >= (window or t))
        for i in range(h):
            s = (q[lo:hi, i] @ k[first:hi, i // per].T * scale).masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[i].to(F64).expand(hi - lo, 1)], 1)
            out[lo:hi, i] = torch.softmax(s, -1)[:, : hi - first] @ v[first:hi, i // per]
    return out


def _ring(x, window, case, cols):
    """Rows of positions x [T, ..., d] as a cache holds them: position p in row p mod ring."""
    max_len = _max_len(case)
    ring = window - 1 + min(PORTION, max_len) if window and window < max_len else max_len
    t = x.shape[0]
    out = torch.zeros(ring, *x.shape[1:-1], cols, dtype=F64, device=x.device)
    lo = max(0, t - ring)
    out[torch.arange(lo, t, device=x.device) % ring, ..., : x.shape[-1]] = x[lo:]
    return out


def _exact_ralasun(case: dict, seed: int):
    w, toks = _weights(case, seed), _tokens(case, seed)
    h, g, d, dv = (case[n] for n in ("heads", "kv_heads", "dim", "vdim"))
    x = _rms(w["embed"][torch.tensor(toks, device="cuda")].to(F64)) * (1 + w["embed.norm"].to(F64))
    t, first, caches = x.shape[0], None, []
    for i in range(case["layers"]):
        m, p = f"l{i}.mix", f"l{i}.mlp"
        q = (_rms(_lin(x, w[f"{m}.q"])) * w[f"{m}.q.norm"].to(F64)).view(t, h, d)
        k = (_rms(_lin(x, w[f"{m}.k"])) * w[f"{m}.k.norm"].to(F64)).view(t, g, d)
        v = _lin(x, w[f"{m}.v"])
        if first is None:
            first = v
        else:
            lam = w[f"{m}.vmix"].to(F64)
            v = (1 - lam) * v + lam * first
        v = v.view(t, g, dv)
        caches += [_ring(c, case["window"], case, (c.shape[-1] + 15) // 16 * 16).transpose(0, 1) for c in (k, v)]
        y = _lin(_attend(q, k, v, d ** -0.5, case["window"]).reshape(t, h * dv), w[f"{m}.o"])
        x = x + _rms(y) * (1 + w[f"l{i}.norm1"].to(F64))
        z = _lin(x, w[f"{p}.router"]) + w[f"{p}.router.b"].to(F64)
        top, ids = torch.topk(z, case["top"], -1)
        share = torch.softmax(top, -1)
        y = _unit(x, *(w[f"{p}.shared.{n}"] for n in ("gate", "up", "down"))) if case["shared_ff"] else torch.zeros_like(x)
        for e in range(case["experts"]):
            row, slot = torch.nonzero(ids == e, as_tuple=True)
            if row.numel():
                y[row] += share[row, slot, None] * _unit(x[row], *(w[f"{p}.e{e}.{n}"] for n in ("gate", "up", "down")))
        x = x + _rms(y) * (1 + w[f"l{i}.norm2"].to(F64))
    return _lin(_rms(x[-1:]) * (1 + w["final.norm"].to(F64)), w["head"]), caches


def _turn(x, cos, sin, interleaved):
    """x [T, ..., d] with cos, sin [T, d / 2]."""
    shape = (x.shape[0],) + (1,) * (x.dim() - 2) + (-1,)
    c, s = cos.view(shape), sin.view(shape)
    half = x.shape[-1] // 2
    a, b = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :half], x[..., half:])
    ya, yb = a * c - b * s, b * c + a * s
    return torch.stack([ya, yb], -1).flatten(-2) if interleaved else torch.cat([ya, yb], -1)


def _exact_rozesun(case: dict, seed: int):
    w, toks = _weights(case, seed), _tokens(case, seed)
    h, d, rot, dv, r = (case[n] for n in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
    x = w["embed"][torch.tensor(toks, device="cuda")].to(F64)
    t, caches = x.shape[0], []
    ang = torch.arange(t, device="cuda", dtype=F64)[:, None] * 1e4 ** (-torch.arange(0, rot, 2, device="cuda", dtype=F64) / rot)
    cos, sin = torch.cos(ang), torch.sin(ang)

    def norm(x, name):
        return _layer_norm(x, w[name], w[f"{name}.b"])

    for i in range(case["layers"]):
        m, near = f"l{i}.mix", i % 2 == 1
        z = norm(x, f"l{i}.norm1")
        ckr = _lin(z, w[f"{m}.dkv"])
        c, kr = _rms(ckr[:, :r]) * w[f"{m}.dkv.norm"].to(F64), _turn(ckr[:, r:], cos, sin, near)
        q = _lin(_rms(_lin(z, w[f"{m}.dq"])) * w[f"{m}.dq.norm"].to(F64), w[f"{m}.uq"]).view(t, h, d + rot)
        q = torch.cat([q[..., :d], _turn(q[..., d:], cos, sin, near)], -1)
        k = torch.cat([_lin(c, w[f"{m}.uk"]).view(t, h, d), kr[:, None].expand(t, h, rot)], -1)
        o = _attend(q, k, _lin(c, w[f"{m}.uv"]).view(t, h, dv), (d + rot) ** -0.5, case["window"] if near else 0, w[f"{m}.sink"] if near else None)
        o = (o * torch.sigmoid(_lin(z, w[f"{m}.g"])).view(t, h, -1)).reshape(t, h * dv)
        rp = (r + 15) // 16 * 16
        row = torch.cat([c, torch.zeros(t, rp - r, dtype=F64, device="cuda"), kr], -1)
        caches.append(_ring(row, case["window"] if near else 0, case, (rp + rot + 31) // 32 * 32))
        x = x + norm(_lin(o, w[f"{m}.o"]), f"l{i}.norm1b")
        y = _unit(norm(x, f"l{i}.norm2"), *(w[f"l{i}.mlp.{n}"] for n in ("gate", "up", "down")))
        x = x + norm(y, f"l{i}.norm2b")
    return _lin(norm(x[-1:], "final.norm"), w["embed"]), caches


def _dequantised(w, name):
    q, s = w[f"{name}.weight"], w[f"{name}.weight_scale_inv"]
    s = s.to(F64).repeat_interleave(128, 0)[: q.shape[0]].repeat_interleave(128, 1)[:, : q.shape[1]]
    return q.to(F32).to(F64) * s


def _dsa_angles(a, t):
    """Rotation angles [t, 32] with the YaRN correction."""
    dim = a.qk_rope_head_dim

    def corr(turns):
        return dim * math.log(a.original_seq_len / (turns * 2 * math.pi)) / (2 * math.log(a.rope_theta))

    f = 1.0 / a.rope_theta ** (torch.arange(0, dim, 2, device="cuda", dtype=F64) / dim)
    lo, hi = max(math.floor(corr(a.beta_fast)), 0), min(math.ceil(corr(a.beta_slow)), dim - 1)
    keep = 1 - ((torch.arange(dim // 2, device="cuda", dtype=F64) - lo) / (hi - lo)).clamp(0, 1)
    f = f / a.rope_factor * (1 - keep) + f * keep
    return torch.arange(t, device="cuda", dtype=F64)[:, None] * f


def _exact_dsa_layer(a, w, li, dense, x, ang, cached):
    """x [S, dim] behind the cached (ki, kv, pe) rows; returns the output and the three caches with the new rows."""
    at, m = f"model.layers.{li}.self_attn", f"model.layers.{li}.mlp"
    s, h, ctx = x.shape[0], a.n_heads, cached[0].shape[0]
    cos, sin = torch.cos(ang[ctx: ctx + s]), torch.sin(ang[ctx: ctx + s])
    z = _rms(x)  # (the gains of these checkpoints are ones)
    kva = z @ _dequantised(w, f"{at}.kv_a_proj_with_mqa").T
    qa = _rms(z @ _dequantised(w, f"{at}.q_a_proj").T)
    kv = torch.cat([cached[1], _rms(kva[:, :512])])
    pe = torch.cat([cached[2], _turn(kva[:, 512:], cos, sin, True)])
    had = torch.ones(1, 1, dtype=F64, device="cuda")
    while had.shape[0] < 128:
        had = torch.cat([torch.cat([had, had], 1), torch.cat([had, -had], 1)])

    def index_rows(v):
        return torch.cat([_turn(v[..., :64], cos, sin, False), v[..., 64:]], -1) @ had * 128 ** -0.5

    ki_new = z @ _dequantised(w, f"{at}.indexer.wk").T
    ki_new = _layer_norm(ki_new, w[f"{at}.indexer.k_norm.weight"], w[f"{at}.indexer.k_norm.bias"])
    ki = torch.cat([cached[0], index_rows(ki_new)])
    iq = index_rows((qa @ _dequantised(w, f"{at}.indexer.wq_b").T).view(s, 64, 128))
    iw = _lin(z, w[f"{at}.indexer.weights_proj.weight"])
    score = torch.einsum("sht,sh->st", torch.relu(torch.einsum("shd,td->sht", iq, ki)), iw)
    t = ki.shape[0]
    late = torch.arange(t, device="cuda")[None] > ctx + torch.arange(s, device="cuda")[:, None]
    score = score.masked_fill(late, -math.inf)
    seen = torch.zeros(s, t, dtype=torch.bool, device="cuda").scatter_(1, torch.topk(score, min(a.index_topk, t), -1)[1], True) & ~late
    q = (qa @ _dequantised(w, f"{at}.q_b_proj").T).view(s, h, 192)
    kvb = _dequantised(w, f"{at}.kv_b_proj").view(h, 256, 512)
    lat = torch.einsum("shd,hdc->shc", q[..., :128], kvb[:, :128])
    scale = 192 ** -0.5 * (0.1 * math.log(a.rope_factor) + 1.0) ** 2
    sc = (torch.einsum("shc,tc->sht", lat, kv) + torch.einsum("shr,tr->sht", _turn(q[..., 128:], cos, sin, True), pe)) * scale
    p = torch.softmax(sc.masked_fill(~seen[:, None], -math.inf), -1)
    o = torch.einsum("shc,hdc->shd", torch.einsum("sht,tc->shc", p, kv), kvb[:, 128:])
    x = x + o.reshape(s, -1) @ _dequantised(w, f"{at}.o_proj").T
    z = _rms(x)

    def unit(z, name):
        g, u = z @ _dequantised(w, f"{name}.gate_proj").T, z @ _dequantised(w, f"{name}.up_proj").T
        return (g * torch.sigmoid(g) * u) @ _dequantised(w, f"{name}.down_proj").T

    if dense:
        return x + unit(z, m), (ki, kv, pe)
    prob = torch.sigmoid(_lin(z, w[f"{m}.gate.weight"]))
    by_group = prob.view(s, a.n_expert_groups, -1)
    keep = torch.topk(torch.topk(by_group, 2, -1)[0].sum(-1), a.n_limited_groups, -1)[1]
    allowed = torch.zeros(s, a.n_expert_groups, dtype=torch.bool, device="cuda").scatter_(1, keep, True)
    ids = torch.topk(by_group.masked_fill(~allowed[..., None], -math.inf).flatten(1), a.n_activated_experts, -1)[1]
    share = prob.gather(1, ids)
    share = share / share.sum(-1, keepdim=True) * a.route_scale
    y = unit(z, f"{m}.shared_experts")
    for e in ids.unique().tolist():
        row, slot = torch.nonzero(ids == e, as_tuple=True)
        y[row] += share[row, slot, None] * unit(z[row], f"{m}.experts.{e}")
    return x + y, (ki, kv, pe)


def _exact_dsa(case: dict, seed: int):
    a, w, toks = _args(case), _weights(case, seed), _tokens(case, seed)
    mtp = case["kind"] == "dsa_mtp"
    ang = _dsa_angles(a, case["ctx"] + len(toks))
    embed = w["model.embed_tokens.weight"]
    x = embed[torch.tensor(toks, device="cuda")].to(F64)
    empty = tuple(torch.zeros(0, d, dtype=F64, device="cuda") for d in (128, 512, 64))
    old = [empty] * 2 if mtp else [tuple(c.to(F64) for c in layer) for layer in _dsa_caches(case, seed)]
    caches = []
    for li in range(2):
        x, rows = _exact_dsa_layer(a, w, li, li == 0, x, ang, old[li])
        caches += rows
    rows_out = (len(toks) - 1) % 4 + 1
    out = {"logits": _lin(_rms(x[-rows_out:]), w["lm_head.weight"])}
    if mtp:
        nxt = embed[torch.tensor(toks[1:] + toks[-1:], device="cuda")].to(F64)
        y, rows = _exact_dsa_layer(a, w, 2, False, _lin(torch.cat([_rms(nxt), _rms(x)], -1), w["model.layers.2.eh_proj.weight"]), ang, empty)
        caches += rows
        return out | {"next": _lin(_rms(y[-rows_out:]), w["lm_head.weight"]), "caches": caches}
    pad = [torch.cat([c, torch.zeros(case["rows"] - c.shape[0], c.shape[1], dtype=F64, device="cuda")]) for c in caches]
    return {"logits": out["logits"].view(1, 1, -1), "caches": pad}


def exact(case: dict, seed: int):
    if case["kind"].startswith("dsa"):
        return _exact_dsa(case, seed)
    logits, caches = (_exact_ralasun if case["kind"] == "ralasun" else _exact_rozesun)(case, seed)
    out = {"logits": logits, "caches": caches}
    if case["sampled"]:
        out["top_logprobs"] = torch.log_softmax(logits, -1).sort(-1, descending=True)[0][:, :256]
    return out
