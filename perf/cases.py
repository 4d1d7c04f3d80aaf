"""What this library is timed on: requests answered through the engine (a step over the prompts, then
single-token steps), prompts alone, and the sampler.

A case is a plain dict.  kind "answer": `batch` prompts whose lengths are spread over [shortest, longest] run in
one step, then `new` single-token steps follow, one token for every sequence, and the slots are given back; `new`
0 is a prompt alone (a long document, or the first token of an answer).  kind "sample": one draw for `rows` rows
of logits with the sampling options a request brings.  Weights are random (no checkpoint is needed to time a
step) with the spread of an initialised network: N(0, 0.02), matrices that write into the residual stream smaller
by sqrt(2 x layers), so that, as in a trained network, one sublayer changes the rows a little and rounding errors
are not amplified from layer to layer.  The tokens fed in are given, not the arg-max of the step before: two
runs whose logits differ in the last bits are then still runs over the same tokens.

A program that serves requests keeps its model and its engine; so does this file, one per model and dtype, while
every `prepare` brings new tokens (or new logits).
"""
from __future__ import annotations

import math
import random
import zlib

import numpy as np
import torch

import zinfer_b200 as z
from zinfer_b200.config.registry import build_model
from zinfer_b200.sampling import Sampler, SamplingParams
from zinfer_b200.weights.loader import load_into

PAGE = 64


# ---------------------------------------------------------------------- models
def _lfm2(hidden, layers, attn_at, heads, ffn):
    return dict(architectures=["Lfm2ForCausalLM"], model_type="lfm2", vocab_size=65536, hidden_size=hidden,
                num_hidden_layers=layers, num_attention_heads=heads, num_key_value_heads=8, max_position_embeddings=128000,
                layer_types=["full_attention" if i in attn_at else "conv" for i in range(layers)],
                block_ff_dim=ffn, block_auto_adjust_ff_dim=False, conv_L_cache=3, conv_bias=False, rope_theta=1000000.0,
                norm_eps=1e-5, tie_word_embeddings=True, eos_token_id=7)


def _zosurax(width, layers, heads, rec_heads, ff, vocab):
    kinds = ["hgrn2", "attention", "attention_2"]
    out = []
    for i in range(layers):
        kind = kinds[i % 3]
        if kind == "hgrn2":
            mixer = {"heads": rec_heads, "dim": 128, "vdim": width // rec_heads}
        else:
            mixer = {"heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 64, "scale": 0.125,
                     "rot": {"base": 10000.0, "dims": 64 if kind == "attention" else 32}}
        out.append({"type": kind, "mixer": mixer, "mlp": {"kind": "dense", "ff": ff}})
    return {"architecture": "Zosurax", "vocab": vocab, "width": width, "max_positions": 4096, "norm": {"eps": 1e-5},
            "layers": out}


def _ponusun(width, layers, heads, window, experts, top, ff, vocab):
    out = []
    for i in range(layers):
        mixer = {"heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": window}}
        if i >= 2 and i % 2 == 0:
            mixer["kv_from"] = i - 1
        mlp = ({"kind": "dense", "ff": 4 * width} if i == 0 else
               {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": experts, "top": top}, "shared": {"ff": ff}})
        out.append({"type": "attention", "mixer": mixer, "mlp": mlp})
    return {"architecture": "Ponusun", "vocab": vocab, "width": width, "max_positions": 4096, "norm": {"eps": 1e-5},
            "canon": {"taps": 3}, "logit_softcap": 20.0, "layers": out}


# The sizes of the repository's benchmark.
MODELS = {
    "lfm2-350m": _lfm2(1024, 16, {2, 5, 8, 10, 12, 14}, 16, 4608),
    "lfm2-1.2b": _lfm2(2048, 16, {2, 5, 8, 10, 12, 14}, 32, 8192),
    "lfm2-2.6b": _lfm2(2048, 30, {2, 6, 10, 14, 18, 21, 24, 27}, 32, 10752),
    "zosurax-w1024": _zosurax(1024, 8, 16, 8, 4096, 32768),
    "zosurax-w2048": _zosurax(2048, 8, 32, 16, 8192, 65536),
    "ponusun-w1024": _ponusun(1024, 8, 16, 512, 16, 2, 1024, 32768),
    "ponusun-w2048": _ponusun(2048, 8, 32, 1024, 16, 2, 2048, 65536),
}
LONGEST = {"lfm2-350m": 16384, "lfm2-1.2b": 32768, "lfm2-2.6b": 8192}           # longest sequence an engine is made for
TOKENS = {"lfm2-350m": 163840, "lfm2-1.2b": 131072}                              # tokens its cache holds
_RESIDUAL = ("out_proj.weight", "w2.weight", "mix.o", ".down")


def _vocab(model):
    d = MODELS[model]
    return d.get("vocab_size") or d["vocab"]


def _n_layers(model):
    d = MODELS[model]
    return d.get("num_hidden_layers") or len(d["layers"])


def _draw_tensor(name, spec, layers):
    """The stored values of one tensor: a function of its name and shape."""
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()))
    shape = spec.stored_shape
    if spec.role == "table":
        return torch.rand(shape[:-1] + (spec.bound,), generator=g, device="cuda").argsort(-1)[..., :shape[-1]].to(torch.int32)
    if spec.init == "unit_interval":
        t = torch.rand(shape, generator=g, device="cuda") * 0.9 + 0.05
    else:
        t = torch.randn(shape, generator=g, device="cuda") * 0.02
        if name.endswith(_RESIDUAL):
            t *= (2 * layers) ** -0.5
        elif name.endswith(".talk"):                # mixed heads: every head mostly itself
            t += torch.eye(shape[0], device="cuda")
        elif name.endswith(".dwa"):                 # depth weights: mostly the last result
            t[-1] += 1.0
        elif spec.init == "abs_normal":
            t = t.abs()
        elif spec.init in ("norm", "one_plus_normal"):
            t += 1.0
    return t.to(torch.bfloat16)


class _Weights(dict):
    """name -> stored tensor, drawn when asked for."""

    def __init__(self, model):
        super().__init__()
        self.specs = build_model(z.config_from_dict(MODELS[model])).weight_specs()
        self.layers = _n_layers(model)

    def __missing__(self, name):
        return _draw_tensor(name, self.specs[name], self.layers)


_ENGINES: dict = {}


def _engine(model, dtype):
    key = (model, dtype)
    if key not in _ENGINES:
        w = _Weights(model)
        found = {n: (torch.int32 if s.role == "table" else torch.bfloat16, s.stored_shape) for n, s in w.specs.items()}
        m = build_model(z.config_from_dict(MODELS[model]))
        load_into(m, lambda n: w[n], found, model, torch.bfloat16 if dtype == "bf16" else torch.float32, "cuda")
        _ENGINES[key] = z.Engine(m, max_batch=64, max_seq_len=LONGEST.get(model, 4096), max_tokens=TOKENS.get(model, 65536),
                                 page_size=PAGE)
    return _ENGINES[key]


# ---------------------------------------------------------------------- cases
def _answer(name, model, batch, shortest, longest, new, dtype="bf16", rows="last"):
    return {"name": name, "kind": "answer", "model": model, "dtype": dtype, "batch": batch, "shortest": shortest,
            "longest": longest, "new": new, "rows": rows}


def _sample(name, rows, vocab, temp, top_k, top_p, min_p):
    return {"name": name, "kind": "sample", "rows": rows, "vocab": vocab, "temp": temp, "top_k": top_k, "top_p": top_p,
            "min_p": min_p}


def listed():
    return [
        # what every generated token of a batch pays behind its step, with the sampling options' defaults
        _sample("sample-8", 8, 65536, 0.8, 40, 0.95, 0.05),
        # the shortest request: a few words in, a few tokens out, the smallest model; launches and host work count
        _answer("short-350m", "lfm2-350m", 1, 11, 11, 8),
        # one user: a question of a page, one token after another
        _answer("answer-1.2b-b1", "lfm2-1.2b", 1, 512, 512, 64),
        # the benchmark's headline batch and prompt lengths
        _answer("answer-1.2b-b8", "lfm2-1.2b", 8, 512, 2048, 64),
        # a loaded server: more rows than the few-row contractions take
        _answer("answer-1.2b-b64", "lfm2-1.2b", 64, 128, 1024, 48),
        # the larger model at a middling batch, odd lengths
        _answer("answer-2.6b-b16", "lfm2-2.6b", 16, 65, 1025, 32),
        # long contexts on the small model: reading the cache counts
        _answer("long-350m-b16", "lfm2-350m", 16, 1024, 8192, 32),
        # time to the first token of the benchmark's prompt
        _answer("prompt-2048", "lfm2-1.2b", 1, 2048, 2048, 0),
        # a document of 32 k tokens, in packed chunks; attention is a third of the work
        _answer("document-32768", "lfm2-1.2b", 1, 32768, 32768, 0),
        # the 32-bit path: logits of every prompt position (scoring, comparing) and a few tokens more
        _answer("fp32-350m", "lfm2-350m", 2, 150, 300, 8, dtype="fp32", rows="all"),
        # recurrences and two kinds of attention
        _answer("zosurax-b8", "zosurax-w2048", 8, 200, 1000, 32),
        # windowed attention, convolutions, experts picked by a table
        _answer("ponusun-b8", "ponusun-w2048", 8, 200, 1000, 32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """Another case of the same ranges: batches of 1 to 64, prompts of 1 to 16,384 tokens, every model."""
    kind = rng.choice(["sample"] + ["prompt"] * 2 + ["answer"] * 6 + ["fp32"])
    if kind == "sample":
        return {k: v for k, v in _sample("", _log_int(rng, 1, 64), rng.choice([32768, 65536]), rng.choice([0.6, 0.8, 1.0]),
                                         rng.choice([20, 40, 100]), rng.choice([0.9, 0.95]), rng.choice([0.0, 0.05])).items()
                if k != "name"}
    if kind == "fp32":
        hi = _log_int(rng, 8, 400)
        c = _answer("", "lfm2-350m", _log_int(rng, 1, 4), max(1, hi // 2), hi, rng.randint(1, 8), dtype="fp32",
                    rows=rng.choice(["last", "all"]))
    elif kind == "prompt":
        n = _log_int(rng, 16, 16384)
        c = _answer("", rng.choice(["lfm2-350m", "lfm2-1.2b"]), 1, n, n, 0)
    else:
        model = rng.choice(["lfm2-350m", "lfm2-1.2b", "lfm2-1.2b", "lfm2-2.6b", "zosurax-w1024", "ponusun-w1024"])
        batch = _log_int(rng, 1, 64)
        hi = _log_int(rng, 8, min(3500, 24000 // batch))
        c = _answer("", model, batch, max(1, hi // rng.choice([1, 2, 4, 8])), hi, rng.randint(4, 48))
    c.pop("name")
    return c


# ---------------------------------------------------------------------- inputs and the pass
def _lengths(case):
    """The prompts' lengths: spread over [shortest, longest], both ends among them, in no order."""
    B, lo, hi = case["batch"], case["shortest"], case["longest"]
    if B == 1:
        return [hi]
    order = random.Random(B * 1000003 + lo * 1009 + hi).sample(range(B), B)
    return [lo + (hi - lo) * i // (B - 1) for i in order]


def _tokens(case, seed):
    rng = np.random.default_rng([int(seed), 17])
    V = _vocab(case["model"])
    prompts = [rng.integers(0, V, size=n).tolist() for n in _lengths(case)]
    return prompts, rng.integers(0, V, size=(case["new"], case["batch"])).tolist()


def _logits(case, seed):
    """Rows like a language model's: a bulk of unlikely tokens and a steep head."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn((case["rows"], case["vocab"]), generator=g, device="cuda") * 2.5


def prepare(case, seed):
    if case["kind"] == "sample":
        params = SamplingParams(temp=case["temp"], top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"], seed=int(seed))
        return {"kind": "sample", "logits": _logits(case, seed), "sampler": Sampler(params, case["vocab"], case["rows"]),
                "requests": list(range(case["rows"]))}
    prompts, forced = _tokens(case, seed)
    want = [list(range(len(p))) for p in prompts] if case["rows"] == "all" else None
    return {"kind": "answer", "engine": _engine(case["model"], case["dtype"]), "prompts": prompts, "forced": forced,
            "want": want, "vocab": _vocab(case["model"])}


def run(state):
    if state["kind"] == "sample":
        return state["sampler"].sample(state["logits"], state["requests"])
    engine, prompts, forced = state["engine"], state["prompts"], state["forced"]
    slots = engine.start(len(prompts))
    try:
        out = {"prompt": engine.step(slots, prompts, want=state["want"], check=False)}
        if forced:
            out["steps"] = torch.empty((len(forced), len(prompts), state["vocab"]), device="cuda")
            for i, tokens in enumerate(forced):
                out["steps"][i].copy_(engine.decode(slots, tokens))      # the engine writes every step's logits to one place
    finally:
        engine.finish(slots)
    return out


# ---------------------------------------------------------------------- what a pass cannot do without
def _layer_work(model):
    """Per layer: (matrix parameters a token meets, parameters a large batch reads, per-token cache values, window,
    query width, recurrent state values)."""
    d = MODELS[model]
    out = []
    if model.startswith("lfm2"):
        D, F, Q, KV = d["hidden_size"], d["block_ff_dim"], d["hidden_size"], 512
        for k in d["layer_types"]:
            if k == "conv":
                out.append((4 * D * D + 3 * D * F, 4 * D * D + 3 * D * F, 0, 0, 0, 2 * D))
            else:
                p = 2 * D * Q + 2 * D * KV + 3 * D * F
                out.append((p, p, 2 * KV, 0, Q, 0))
        return out
    D = d["width"]
    for L in d["layers"]:
        m, f = L["mixer"], L["mlp"]
        if L["type"] == "hgrn2":
            p, kv, win, q, st = 2 * D * m["heads"] * m["dim"] + 2 * D * D, 0, 0, 0, m["heads"] * m["dim"] * m["vdim"]
        else:
            q, kvw = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
            p = 2 * D * q + (0 if "kv_from" in m else 2 * D * kvw)
            kv, win, st = 2 * kvw, (m.get("mask") or {}).get("size", 0), 0
        if f["kind"] == "dense":
            active = every = 2 * D * f["ff"]
        else:
            one = 3 * D * f["expert"]["ff"]
            active = one * f["router"]["top"] + 3 * D * f["shared"]["ff"]
            every = one * f["router"]["experts"] + 3 * D * f["shared"]["ff"]
        out.append((p + active, p + every, kv, win, q, st))
    return out


def work(case):
    """Bytes: the weights once for the prompts (a chunk of prompt tokens meets all of them) and once per single-token
    step, which cannot start before the token of the step before is known; keys and values written once and read by
    every later step; the logits.  FLOPs: 2 per matrix parameter and token met, 4 x query width per attended pair."""
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n + 4 * case["rows"], "flops": 0}
    size = 2 if case["dtype"] == "bf16" else 4
    lens, new, B, V = _lengths(case), case["new"], case["batch"], _vocab(case["model"])
    d = MODELS[case["model"]]
    D = d.get("hidden_size") or d["width"]
    total, bytes_, flops = sum(lens), 0.0, 0.0
    head_rows = (total if case["rows"] == "all" else B) + new * B
    for active, every, kv, win, q, state in _layer_work(case["model"]):
        experts = every - active
        per_step = active + min(experts, experts * (B - 1) / 7.0) if experts else active    # 8 x 2 of 16 experts: all of them
        bytes_ += size * ((every if total >= 8 else per_step) + new * per_step)
        flops += 2.0 * active * (total + new * B)
        if q:
            pairs = 0
            for n in lens:
                w = win or n + new + 1
                pairs += sum(min(i + 1, w) for i in range(n + new)) if n + new < 4096 else (n + new) * (n + new + 1) / 2
                bytes_ += size * kv * (n + new + sum(min(n + i + 1, w) for i in range(new)))
            flops += 4.0 * q * pairs
        bytes_ += 4.0 * state * B * (1 + 2 * new)
    bytes_ += size * V * D * (1 + new) + 4.0 * V * head_rows
    flops += 2.0 * V * D * head_rows
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Measured against `exact`: 0.5e-2 (8 layers) to 1.8e-2 (30 layers) in bfloat16, from the rounding of the rows that
    enter every contraction; two implementations that round at other places differ by up to sqrt(2) of that.  In
    32 bits 6e-6 with sums in k order."""
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "fp32":
        return {"rel": 2.5e-5}
    return {"rel": 3e-2}


# ---------------------------------------------------------------------- the same in 64 bits, plain torch
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, base, n_rot, interleaved):
    """x [T, heads, d], positions 0..T-1."""
    T = x.shape[0]
    half = n_rot // 2
    inv = float(base) ** (-torch.arange(half, dtype=torch.float64, device=x.device) * 2.0 / n_rot)
    ang = torch.arange(T, dtype=torch.float64, device=x.device)[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = (slice(0, n_rot, 2), slice(1, n_rot, 2)) if interleaved else (slice(0, half), slice(half, n_rot))
    y = x.clone()
    y[..., a] = x[..., a] * c - x[..., b] * s
    y[..., b] = x[..., b] * c + x[..., a] * s
    return y


def _attend(q, k, v, scale, window=0, r1=None, r2=None, talk=None):
    """q [T, H, d], k and v [T, G, d]; query blocks keep the scores small."""
    T, H, d = q.shape
    G = k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    kk, vv = k.permute(1, 2, 0), v.permute(1, 0, 2)
    block = max(64, min(1024, int(1.5e9 // (8 * H * T))))
    for lo in range(0, T, block):
        hi = min(T, lo + block)
        s = torch.matmul(q[lo:hi].reshape(hi - lo, G, H // G, d).permute(1, 2, 0, 3), kk[:, None, :, :hi]) * scale
        s = s.reshape(H, hi - lo, hi)
        dist = torch.arange(lo, hi, device=q.device)[:, None] - torch.arange(hi, device=q.device)
        if r1 is not None:
            s -= r1[:, None, None] * torch.log1p(r2[:, None, None] * dist.clamp(min=0))
        s.masked_fill_((dist < 0) | (dist >= window) if window else dist < 0, -math.inf)
        s = torch.softmax(s, -1)
        if talk is not None:
            s = torch.einsum("hg,gij->hij", talk, s)
        o = torch.matmul(s.reshape(G, H // G, hi - lo, hi), vv[:, None, :hi])
        out[lo:hi] = o.reshape(H, hi - lo, -1).permute(1, 0, 2)
    return out.reshape(T, -1)


def _silu(x):
    return x * torch.sigmoid(x)


def _shifted(x, cuts, by):
    """Row t - by of the same sequence, 0 before its start; `cuts` are the sequences' bounds in the packed rows."""
    y = torch.zeros_like(x)
    for a, b in zip(cuts, cuts[1:]):
        if b - a > by:
            y[a + by:b] = x[a:b - by]
    return y


def _per_sequence(cuts, f, *rows):
    return torch.cat([f(*(r[a:b] for r in rows)) for a, b in zip(cuts, cuts[1:])])


def _exact_lfm2(d, W, x, cuts, tokens):
    eps, H, G = d["norm_eps"], d["num_attention_heads"], 8
    hd = d["hidden_size"] // H
    for i, kind in enumerate(d["layer_types"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * W(p + "operator_norm.weight")
        if kind == "conv":
            b, c, u = (h @ W(p + "conv.in_proj.weight").T).chunk(3, -1)
            u = b * u
            taps = W(p + "conv.conv.weight").reshape(-1, d["conv_L_cache"])
            n = taps.shape[1]
            y = sum(taps[:, j] * _shifted(u, cuts, n - 1 - j) for j in range(n))
            x = x + (c * y) @ W(p + "conv.out_proj.weight").T
        else:
            a = p + "self_attn."
            q, k, v = ((h @ W(a + n + "_proj.weight").T).reshape(len(h), -1, hd) for n in "qkv")
            q, k = _rms(q, eps) * W(a + "q_layernorm.weight"), _rms(k, eps) * W(a + "k_layernorm.weight")

            def attend(q, k, v):
                return _attend(_rotate(q, d["rope_theta"], hd, False), _rotate(k, d["rope_theta"], hd, False), v, hd ** -0.5)

            x = x + _per_sequence(cuts, attend, q, k, v) @ W(a + "out_proj.weight").T
        h = _rms(x, eps) * W(p + "ffn_norm.weight")
        f = p + "feed_forward."
        x = x + (_silu(h @ W(f + "w1.weight").T) * (h @ W(f + "w3.weight").T)) @ W(f + "w2.weight").T
    return lambda r: (_rms(r, eps) * W("model.embedding_norm.weight")) @ W("model.embed_tokens.weight").T, x


def _hgrn2(q, f, v, cuts):
    """S <- diag(f) S + (1 - f) v^T, o = S^T q, all sequences side by side."""
    lens = [b - a for a, b in zip(cuts, cuts[1:])]
    S = torch.zeros((len(lens), *q.shape[1:], v.shape[2]), dtype=q.dtype, device=q.device)
    out = torch.empty_like(v)
    base = torch.tensor(cuts[:-1], device=q.device)
    for t in range(max(lens)):
        live = [b for b, n in enumerate(lens) if n > t]
        at = base[live] + t
        Sl = S[live]
        ft = f[at]
        Sl = ft[..., None] * Sl + (1 - ft)[..., None] * v[at][:, :, None, :]
        S[live] = Sl
        out[at] = torch.einsum("bhde,bhd->bhe", Sl, q[at])
    return out


def _exact_zosurax(d, W, x, cuts, tokens):
    eps = d["norm"]["eps"]
    for i, L in enumerate(d["layers"]):
        p, m = f"l{i}.", L["mixer"]
        h = _rms(x, eps) * W(p + "norm1")
        h = h + (_shifted(h, cuts, 1) - h) * W(p + "shift")
        a = p + "mix."
        T, hd = len(h), m["dim"]
        if L["type"] == "hgrn2":
            H = m["heads"]
            low = W(a + "lower").reshape(H, hd)
            f = low + (1 - low) * torch.sigmoid(h @ W(a + "f").T + W(a + "f.b")).reshape(T, H, hd)
            o = _hgrn2(_silu(h @ W(a + "q").T).reshape(T, H, hd), f, (h @ W(a + "v").T).reshape(T, H, -1), cuts)
            y = (_rms(o, eps) * W(a + "norm")).reshape(T, -1) @ W(a + "o").T
        else:
            talk, rot = L["type"] == "attention_2", m["rot"]
            q, k, v = ((h @ W(a + n).T).reshape(T, -1, hd) for n in "qkv")
            if not talk:
                q, k = _rms(q, eps) * W(a + "q.norm"), _rms(k, eps) * W(a + "k.norm")

            def attend(q, k, v):
                q, k = (_rotate(r, rot["base"], rot["dims"], talk) for r in (q, k))
                if talk:
                    q, k = _rms(q, eps), _rms(k, eps)
                return _attend(q, k, v, m["scale"], talk=W(a + "talk") if talk else None)

            y = _per_sequence(cuts, attend, q, k, v) @ W(a + "o").T
        x = x + y * W(p + "ls1")
        u = torch.relu((_rms(x, eps) * W(p + "norm2")) @ W(p + "mlp.up").T)
        x = x + ((u * u) @ W(p + "mlp.down").T) * W(p + "ls2")
    return lambda r: (_rms(r, eps) * W("final.norm")) @ W("embed").T, x


def _exact_ponusun(d, W, x, cuts, tokens):
    eps, cap = d["norm"]["eps"], d["logit_softcap"]
    at = torch.cat([torch.arange(b - a, device="cuda") for a, b in zip(cuts, cuts[1:])])
    x = x + W("pos")[at]
    results, kv_of = [x], {}
    for i, L in enumerate(d["layers"]):
        p, m = f"l{i}.", L["mixer"]
        c = W(p + "canon1")
        n = c.shape[1]
        h = x + sum(c[:, j] * _shifted(x, cuts, n - 1 - j) for j in range(n))
        a = p + "mix."
        T, hd = len(h), m["dim"]
        q = (_rms(h @ W(a + "q").T, eps) * W(a + "q.norm")).reshape(T, -1, hd)
        if "kv_from" in m:
            k, v = kv_of[m["kv_from"]]
        else:
            k = (_rms(h @ W(a + "k").T, eps) * W(a + "k.norm")).reshape(T, -1, hd)
            v = (h @ W(a + "v").T).reshape(T, -1, hd)
            kv_of[i] = k, v
        r1, r2 = W(a + "r1"), W(a + "r2")
        y = _per_sequence(cuts, lambda q, k, v: _attend(q, k, v, m["scale"], m["mask"]["size"], r1, r2), q, k, v)
        x = x + _rms(y @ W(a + "o").T, eps) * W(p + "norm1")
        if L["mlp"]["kind"] == "dense":
            f = torch.nn.functional.gelu(x @ W(p + "mlp.up").T) @ W(p + "mlp.down").T
        else:
            def gated(x, e):
                return (_silu(x @ W(e + "gate").T) * (x @ W(e + "up").T)) @ W(e + "down").T

            picks = W(p + "mlp.table")[tokens]
            f = torch.sigmoid(x @ W(p + "mlp.shared.sg").reshape(-1))[:, None] * gated(x, p + "mlp.shared.")
            for e in range(L["mlp"]["router"]["experts"]):
                mine = (picks == e).any(-1).nonzero().reshape(-1)
                if len(mine):
                    f[mine] += gated(x[mine], f"{p}mlp.e{e}.") / picks.shape[1]
        x = x + _rms(f, eps) * W(p + "norm2")
        results.append(x)
        w = W(p + "dwa").reshape(-1)
        x = sum(w[j] * results[j] for j in range(len(results)))
    return lambda r: cap * torch.tanh((_rms(r, eps) * W("final.norm")) @ W("head").T / cap), x


def exact(case, seed):
    """Whole sequences (prompt and the tokens fed in behind it) in 64 bits without a cache; the rows that `run` returns."""
    if case["kind"] == "sample":
        return None
    d, w = MODELS[case["model"]], _Weights(case["model"])

    def W(name):
        t = w[name]
        return t.double() if t.is_floating_point() else t.long()

    prompts, forced = _tokens(case, seed)
    B, new = case["batch"], case["new"]
    seqs = [p + [forced[i][b] for i in range(new)] for b, p in enumerate(prompts)]
    cuts = [0, *np.cumsum([len(s) for s in seqs]).tolist()]
    tokens = torch.tensor([t for s in seqs for t in s], device="cuda")
    arch = case["model"].split("-")[0]
    x = W("model.embed_tokens.weight" if arch == "lfm2" else "embed")[tokens]
    head, x = {"lfm2": _exact_lfm2, "zosurax": _exact_zosurax, "ponusun": _exact_ponusun}[arch](d, W, x, cuts, tokens)
    if case["rows"] == "all":
        first = [cuts[b] + i for b, p in enumerate(prompts) for i in range(len(p))]
    else:
        first = [cuts[b] + len(p) - 1 for b, p in enumerate(prompts)]
    later = [cuts[b] + len(prompts[b]) + i for i in range(new) for b in range(B)]
    out = {"prompt": head(x[first])}
    if new:
        out["steps"] = head(x[later]).reshape(new, B, -1)
    return out
