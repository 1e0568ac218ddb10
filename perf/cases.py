"""Performance cases of the framework: the calls a serving program, an embedding service or a scoring job makes, at the sizes of the
models that the benchmark and the tests use (few layers of each, so that a model fits beside others and a 64-bit result stays
affordable).  Every pass goes through the public Python entry points with host token ids in and host logits / embeddings out."""
from __future__ import annotations

import math

import numpy as np
import torch

from fastllm_b200 import models

# ---- models -----------------------------------------------------------------------------------------------------------------------
# (class, hidden, intermediate, vocabulary, query heads, key/value heads, norm eps, rope theta): the Llama-family sizes of the benchmark
LLAMA_FAMILY = {
    "tinyllama": (models.LlamaWithConfig, 2048, 5632, 32000, 32, 4, 1e-5, 1e4),
    "mistral7b": (models.MistralWithConfig, 4096, 14336, 32000, 32, 8, 1e-5, 1e4),
    "qwen25_7b": (models.QwenWithConfig, 3584, 18944, 152064, 28, 4, 1e-6, 1e6),
    "mixtral8x7b": (models.MixtralWithConfig, 4096, 14336, 32000, 32, 8, 1e-5, 1e6),
}
EXPERTS, TOP = 8, 2
LAYERED_VOCAB = 32000
MAX_SEQ = 4096              # tokens a serving cache holds per sequence
FEED_FORWARD = {1024: 2816, 2048: 5632, 4096: 14336}     # hidden width of a dense feed-forward at each layered width


def _nifunex(W):
    """gated linear attention and windowed latent attention in turn, experts with a shared one"""
    H, ff = W // 128, FEED_FORWARD[W]
    mlp = {"kind": "moe", "expert": {"ff": ff, "limit": 7.0}, "router": {"experts": EXPERTS, "top": TOP}, "shared": {"ff": ff, "limit": 7.0}}
    return {"layers": [
        {"type": "gla", "mixer": {"heads": H, "dim": 128, "vdim": 128, "tau": 16.0}, "mlp": mlp},
        {"type": "latent_attention", "mixer": {"heads": H, "dim": 96, "rot_dim": 32, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5,
                                               "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 32}}, "mlp": mlp}]}


def _rofetar(W):
    """gated delta rule, grouped-query attention with sink and score cap, Mamba-2; dense gelu feed-forwards"""
    H, mlp = W // 128, {"kind": "dense", "ff": FEED_FORWARD[W]}
    rot = {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}}
    return {"layers": [
        {"type": "delta", "mixer": {"heads": H, "kv_heads": H // 2, "dim": 128, "vdim": 128, "conv": 4}, "mlp": mlp},
        {"type": "attention", "mixer": {"heads": H, "kv_heads": H // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0, "rot": rot}, "mlp": mlp},
        {"type": "mamba2", "mixer": {"heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": H // 4, "norm_groups": 1, "conv": 4}, "mlp": mlp}]}


def _medulorn(W):
    """windowed attention with kept first tokens beside lightning attention, chunk-masked attention; experts with a shared one"""
    H, ff = W // 128, FEED_FORWARD[W] // 2
    mlp = {"kind": "moe", "expert": {"ff": ff, "limit": 7.0}, "router": {"experts": EXPERTS, "top": TOP}, "shared": {"ff": ff, "limit": 7.0}}
    rot = {"base": 500000.0, "dims": 128}
    left = {"heads": H, "kv_heads": H // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024, "keep_first": 4}, "rot": rot}
    right = {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + 5 * h / max(1, H - 1)) for h in range(H)]}
    return {"postln_alpha": 1.0, "embedding": {"scale": 1.0}, "logit_softcap": 50.0, "layers": [
        {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 0.5, "right_scale": 0.5}, "mlp": mlp},
        {"type": "attention", "mixer": {"heads": H, "kv_heads": H // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 8192}, "rot": rot}, "mlp": mlp}]}


def _tufazen(W):
    """latent attention with a dense feed-forward, grouped-query attention with experts, both sublayers in parallel; token vectors"""
    H, ff = W // 128, FEED_FORWARD[W]
    return {"logit_scale": 1.0, "token_side": {"dim": 128},
            "embedding": {"bigram": {"buckets": LAYERED_VOCAB - 3, "mul_prev": 1000003, "mul_cur": 31}}, "layers": [
        {"type": "latent_attention", "mlp": {"kind": "dense", "ff": ff, "limit": 7.0},
         "mixer": {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": W * 3 // 8, "scale": 192 ** -0.5, "rot": {"base": 10000.0, "dims": 64}}},
        {"type": "attention", "mlp": {"kind": "moe", "expert": {"ff": ff // 2}, "shared": {"ff": ff // 2},
                                      "router": {"experts": EXPERTS, "top": TOP, "groups": {"count": 4, "keep": 2}}},
         "mixer": {"heads": H, "kv_heads": H // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
                   "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}}]}


LAYERED = {"nifunex": (models.NifunexWithConfig, _nifunex), "rofetar": (models.RofetarWithConfig, _rofetar),
           "medulorn": (models.MedulornWithConfig, _medulorn), "tufazen": (models.TufazenWithConfig, _tufazen)}


def _layered_config(family, width):
    return {"architecture": family.capitalize(), "vocab": LAYERED_VOCAB, "width": width, "norm": {"eps": 1e-6}, **LAYERED[family][1](width)}


# ---- the cases --------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one search query through the all-MiniLM-L6-v2 encoder: the smallest call, an interactive one
        {"name": "embed_query", "work": "embed", "batch": 1, "tokens": 19},
        # indexing: a full batch of 128-token passages through the encoder
        {"name": "embed_batch", "work": "embed", "batch": 256, "tokens": 128},
        # a single chat: one token per call at a 2k context, Mistral-7B layers
        {"name": "chat_decode", "work": "decode", "model": "mistral7b", "layers": 4, "batch": 1, "context": 2048, "ragged": False},
        # static batch of eight chats
        {"name": "batch_decode", "work": "decode", "model": "mistral7b", "layers": 4, "batch": 8, "context": 2048, "ragged": False},
        # a loaded server: 64 sequences of their own lengths in one step
        {"name": "server_decode", "work": "decode", "model": "mistral7b", "layers": 2, "batch": 64, "context": 2048, "ragged": True},
        # a loaded mixture-of-experts server
        {"name": "moe_decode", "work": "decode", "model": "mixtral8x7b", "layers": 1, "batch": 32, "context": 500, "ragged": True},
        # reading a long document, Qwen2.5-7B layers with their vocabulary: the largest call
        {"name": "long_prefill", "work": "prefill", "model": "qwen25_7b", "layers": 2, "tokens": 4096},
        # a prompt through a layered model with recurrent and latent-attention layers and experts
        {"name": "nifunex_prefill", "work": "step", "model": "nifunex", "width": 2048, "dtype": "bf16", "decoding": 0, "context": 0, "tokens": 1531},
        # a prompt through delta-rule, attention and state-space layers
        {"name": "rofetar_prefill", "work": "step", "model": "rofetar", "width": 4096, "dtype": "bf16", "decoding": 0, "context": 0, "tokens": 2048},
        # continuous batching: a portion of one prompt beside seven sequences that decode
        {"name": "medulorn_mixed", "work": "step", "model": "medulorn", "width": 2048, "dtype": "bf16", "decoding": 7, "context": 700, "tokens": 333},
        # eight decoding sequences of a layered model
        {"name": "tufazen_decode", "work": "step", "model": "tufazen", "width": 4096, "dtype": "bf16", "decoding": 8, "context": 2000, "tokens": 0},
        # the exact mode, as a trace is replayed for comparison: a short prompt with every product in 32 bits or better
        {"name": "rofetar_exact", "work": "step", "model": "rofetar", "width": 1024, "dtype": "f32", "decoding": 0, "context": 0, "tokens": 203},
    ]


def _spread(rng, lo, hi):
    """a whole number, even over the logarithm"""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["embed", "decode", "decode", "prefill", "step", "step", "step"])
    if kind == "embed":
        tokens = _spread(rng, 4, 512)
        return {"work": kind, "batch": _spread(rng, 1, min(256, 32768 // tokens)), "tokens": tokens}
    if kind == "decode":
        model = rng.choice(sorted(LLAMA_FAMILY))
        moe = model == "mixtral8x7b"
        return {"work": kind, "model": model, "layers": 1 if moe else rng.randint(1, 4 if model == "tinyllama" else 2),
                "batch": _spread(rng, 1, 32 if moe else 64), "context": _spread(rng, 16, 500 if moe else 2000), "ragged": rng.random() < 0.5}
    if kind == "prefill":
        return {"work": kind, "model": rng.choice(["tinyllama", "mistral7b", "qwen25_7b"]), "layers": rng.randint(1, 2), "tokens": _spread(rng, 8, 2048)}
    model = rng.choice(sorted(LAYERED))
    dtype = "f32" if rng.random() < 0.15 else "bf16"
    width = 1024 if dtype == "f32" else rng.choice([1024, 2048])
    decoding = rng.choice([0, 0, _spread(rng, 1, 8)])
    tokens = _spread(rng, 8, 203 if dtype == "f32" else 1531) if decoding == 0 or rng.random() < 0.5 else 0
    return {"work": kind, "model": model, "width": width, "dtype": dtype, "decoding": decoding,
            "context": _spread(rng, 16, 100 if dtype == "f32" else 1000) if decoding else 0, "tokens": tokens}


def _std(width):
    return width ** -0.5


def _tokens(seed, n, vocab):
    """ids spread over the vocabulary (the first few are special)"""
    return np.random.default_rng(seed).integers(3, vocab, n).astype(np.uint32)


def _lengths(case):
    """what every sequence of a decode step holds already: the context, or lengths from a quarter of it up to it"""
    b, c = case["batch"], case["context"]
    if not case["ragged"]:
        return [c] * b
    lo = max(1, c // 4)
    return [lo + (c - lo) * (i * 7 % b) // max(1, b - 1) for i in range(b)]


# ---- preparation: weights, caches and token ids -----------------------------------------------------------------------------------
def _small_tensors(config, family, seed):
    """the per-head and per-channel constants of a layered model, in the ranges trained models have them (the synthetic fill would
    leave them all alike); every value is a bf16 one.  name -> f32 array"""
    rng = np.random.default_rng(seed)
    out = {}

    def put(name, a):
        out[name] = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).bfloat16().float().numpy()
    for i, l in enumerate(config["layers"]):
        m, p = l["mixer"], f"l{i}.mix."
        if l["type"] == "delta":
            put(p + "A_log", rng.uniform(-3.0, 0.5, m["heads"]))
            put(p + "dt_bias", rng.uniform(-3.0, 0.0, m["heads"]))
            for n, rows in (("q", m["kv_heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]), ("v", m["heads"] * m["vdim"])):
                put(p + n + ".conv", rng.normal(0.0, 0.5, (rows, m["conv"])))
        elif l["type"] == "mamba2":
            channels = m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
            put(p + "A_log", rng.uniform(-2.0, 0.5, m["heads"]))
            put(p + "dt_bias", rng.uniform(-3.0, 0.0, m["heads"]))
            put(p + "conv", rng.normal(0.0, 0.5, (channels, m["conv"])))
        elif l["type"] == "parallel":
            put(p + "left.sink", rng.normal(0.0, 1.0, m["left"]["heads"]))
        elif family == "tufazen" and l["type"] == "attention":
            put(p + "sink", rng.normal(0.0, 1.0, m["heads"]))
        if family == "medulorn":
            put(f"l{i}.shift", rng.uniform(0.05, 0.95, config["width"]))
    return out


def _layered_model(family, width, dtype, seed):
    cls, config = LAYERED[family][0], _layered_config(family, width)
    small = _small_tensors(config, family, seed)

    class WithConstants(cls):
        @classmethod
        def config_tensors(c, cfg):
            yield from cls.config_tensors(cfg)
            yield from small.items()
    model, _ = WithConstants.initialize_model(config, None, dtype, 0, random_seed=seed, std=_std(width))
    return model


def _llama_model(case, seed):
    cls, H, I, V, heads, kv, eps, theta = LLAMA_FAMILY[case["model"]]
    cfg = models.ConfigFile(H, I, V, case["layers"], heads, kv, eps, theta, MAX_SEQ,
                            num_local_experts=EXPERTS if case["model"] == "mixtral8x7b" else 0, num_experts_per_tok=TOP)
    model, _ = cls.initialize_model(cfg, None, "bf16", 0, random_seed=seed, std=_std(H))
    return model


def _llama_decode_tokens(case, seed):
    """-> (one shared prefix that the sequences hold more or less of, the token each sequence is fed)"""
    V = LLAMA_FAMILY[case["model"]][3]
    ids = _tokens(seed + 1, max(_lengths(case)) + case["batch"], V)
    return ids[:-case["batch"]], ids[-case["batch"]:]


def _step_tokens(case, seed):
    """-> (what each decoding sequence holds, the token each is fed, the portion of a prompt beside them)"""
    n, c = case["decoding"], case["context"]
    lengths = [max(1, c - (c // 10) * i // max(1, n)) for i in range(n)]
    ids = _tokens(seed + 1, sum(lengths) + n + case["tokens"], LAYERED_VOCAB)
    held, at = [], 0
    for k in lengths:
        held.append(ids[at:at + k])
        at += k
    return held, ids[at:at + n], ids[at + n:]


def prepare(case, seed):
    s = {"case": case}
    if case["work"] == "embed":
        s["model"] = models.MiniLMModel(models.BertConfig(), None, 0, random_seed=seed)
        s["ids"] = _tokens(seed + 1, case["batch"] * case["tokens"], 30522).reshape(case["batch"], case["tokens"])
    elif case["work"] == "prefill":
        s["model"] = _llama_model(case, seed)
        s["cache"] = models.DeviceCache(s["model"].dev, 1, MAX_SEQ)
        s["ids"] = _tokens(seed + 1, case["tokens"], LLAMA_FAMILY[case["model"]][3])[None]
    elif case["work"] == "decode":
        s["model"] = _llama_model(case, seed)
        s["cache"] = models.DeviceCache(s["model"].dev, case["batch"], MAX_SEQ)
        s["prefix"], s["next"] = _llama_decode_tokens(case, seed)
        _read_prompts(s)
    else:
        s["model"] = _layered_model(case["model"], case["width"], case["dtype"], seed)
        n = case["decoding"] + (1 if case["tokens"] else 0)
        s["cache"] = s["model"].new_device_cache(max_batch=n, max_seq=MAX_SEQ, pool_tokens=n * MAX_SEQ)
        s["held"], s["next"], s["portion"] = _step_tokens(case, seed)
        _read_prompts(s)
    return s


def _read_prompts(s):
    """the sequences of a decode step read what they hold; done again when one of them has filled its share of the cache"""
    case, cache = s["case"], s["cache"]
    if case["work"] == "decode":
        cache.reset()
        s["lengths"] = _lengths(case)
        if case["ragged"]:
            for i, k in enumerate(s["lengths"]):
                cache.forward_slots([i], s["prefix"][None, :k], [0])
        else:
            cache.forward(np.tile(s["prefix"][None], (case["batch"], 1)), 0)
    else:
        s["lengths"] = [len(h) for h in s["held"]]
        for i, h in enumerate(s["held"]):
            cache.slot_reset(i)
            cache.forward_ragged([i], [h], [[]])


def run(state):
    case = state["case"]
    if case["work"] == "embed":
        return state["model"].embed_ids(state["ids"])
    cache = state["cache"]
    if case["work"] == "prefill":
        cache.reset()
        return cache.forward(state["ids"], 0)
    if state["lengths"] and max(state["lengths"]) >= MAX_SEQ:
        _read_prompts(state)
    at = state["lengths"]
    state["lengths"] = [k + 1 for k in at]
    if case["work"] == "decode":
        if case["ragged"]:
            return cache.forward_slots(range(len(at)), state["next"][:, None], at)
        return cache.forward(state["next"][:, None], at[0])
    slots, lists = list(range(len(at))), [[t] for t in state["next"]]
    if case["tokens"]:
        cache.slot_reset(len(at))
        slots.append(len(at))
        lists.append(state["portion"])
    return cache.forward_ragged(slots, lists)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def _hit(rows):
    """experts that `rows` tokens are expected to choose"""
    return EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** rows)


def _layered_sizes(case):
    """per layer: (weights always read, weights of one expert, cached values per token and keys' reach, floats of a recurrent state,
    multiply-adds per token and visible key, multiply-adds per token of a recurrence)"""
    out = []
    W = case["width"]
    for l in _layered_config(case["model"], W)["layers"]:
        mlp, always, kv, reach, state, per_key, rec = l["mlp"], 0, 0, 0, 0, 0, 0
        for kind, m in ((l["type"], l["mixer"]),) if l["type"] != "parallel" else (("attention", l["mixer"]["left"]), ("lightning", l["mixer"]["right"])):
            H = m["heads"]
            if kind == "attention":
                shared = case["model"] == "tufazen"         # values are the keys before they turn; a gate per channel
                always += W * (H * m["dim"] * (3 if shared else 2) + m["kv_heads"] * m["dim"] * (1 if shared else 2))
                kv += m["kv_heads"] * ((m["dim"] + m["rot"]["dims"]) if shared else 2 * m["dim"])
                reach, per_key = (m.get("mask") or {}).get("size") or 1 << 30, H * 2 * m["dim"]
            elif kind == "latent_attention":
                C, R, D, Dv, Q = m["kv_rank"], m["rot_dim"], m["dim"], m["vdim"], m.get("q_rank", 0)
                always += W * (C + R) + H * C * (D + Dv) + W * H * Dv + (W * Q + Q * H * (D + R) + W * H if Q else W * H * (D + R))
                kv += C + R
                reach, per_key = (m.get("mask") or {}).get("size") or 1 << 30, H * (D + R + Dv)
            elif kind == "mamba2":
                inner, gn = H * m["vdim"], m["groups"] * m["state"]
                always += W * (3 * inner + 2 * gn + H)
                state, rec = state + H * m["state"] * m["vdim"], rec + 2 * H * m["state"] * m["vdim"]
            else:
                G = m.get("kv_heads", H)
                always += W * (2 * G * m["dim"] + 3 * H * m["vdim"]) + (W * 2 * H if kind == "delta" else 0)
                state, rec = state + H * m["dim"] * m["vdim"], rec + (3 if kind == "delta" else 2) * H * m["dim"] * m["vdim"]
        F = mlp["expert"]["ff"] if mlp["kind"] == "moe" else 0
        always += 3 * W * (mlp["ff"] if mlp["kind"] == "dense" else mlp["shared"]["ff"])
        out.append((always, 3 * W * F, kv, reach, state, per_key, rec))
    return out


def work(case):
    if case["work"] == "embed":
        H, I, L, b, t = 384, 1536, 6, case["batch"], case["tokens"]
        per_layer = 4 * H * H + 2 * H * I
        return {"bytes": 2 * L * per_layer + 2 * b * t * H + 4 * b * H, "flops": 2.0 * b * t * L * (per_layer + 2 * t * H)}
    if case["work"] != "step":
        _, H, I, V, heads, kv, _, _ = LLAMA_FAMILY[case["model"]]
        d = H // heads
        moe = case["model"] == "mixtral8x7b"
        attn, ff = H * d * (2 * heads + 2 * kv), 3 * H * I
        if case["work"] == "decode":
            rows, keys, wanted = case["batch"], sum(_lengths(case)) + case["batch"], case["batch"]
            read = keys
        else:
            rows, wanted = case["tokens"], 1
            keys, read = rows * (rows + 1) // 2, rows
        weights = case["layers"] * (attn + ff * (_hit(rows) if moe else 1)) + V * H
        active = case["layers"] * (attn + ff * (TOP if moe else 1))
        return {"bytes": 2.0 * weights + 2 * case["layers"] * 2 * kv * d * read + 4 * wanted * V,
                "flops": 2.0 * (rows * active + wanted * V * H) + 4.0 * case["layers"] * keys * heads * d}
    W, size = case["width"], 2 if case["dtype"] == "bf16" else 4
    held = [len(h) for h in _step_tokens(case, 0)[0]]
    rows, wanted = len(held) + case["tokens"], len(held) + (1 if case["tokens"] else 0)
    moved, flops = 2.0 * LAYERED_VOCAB * W + 4.0 * wanted * LAYERED_VOCAB, 2.0 * wanted * LAYERED_VOCAB * W
    for always, expert, kv, reach, state, per_key, rec in _layered_sizes(case):
        T = case["tokens"]
        seen = sum(min(k + 1, reach) for k in held) + sum(min(k + 1, reach) for k in range(T))
        moved += 2.0 * (always + expert * _hit(rows)) + size * kv * (sum(min(k + 1, reach) for k in held) + T) + 4.0 * state * (2 * len(held) + (1 if T else 0))
        flops += 2.0 * rows * (always + TOP * expert) + 2.0 * seen * per_key + 2.0 * rows * rec
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """about four times what the results of one precision are from 64 bits: the Llama family and the encoder keep keys, values (and the
    encoder its activations) in bf16, which shows in the logits as 3e-3 to 5e-3; the layered models' norms behind every sublayer leave
    1e-5 to 1e-3 of it; the exact mode is at 2e-7 to 3e-7"""
    if case["work"] != "step":
        return {"rel": 2e-2}
    return {"rel": 1.2e-6 if case["dtype"] == "f32" else 4e-3}


# ---- the same results in 64 bits ----------------------------------------------------------------------------------------------------
GOLDEN, M64 = 0x9E3779B97F4A7C15, (1 << 64) - 1
F64 = torch.float64


def _signed(v):
    v &= M64
    return v - (1 << 64) if v >> 63 else v


def _mix(z):
    z &= M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


class _Weights:
    """the synthetic weights of a seed (a counter-based hash of the tensor's name and the element's number, four 16-bit fields summed,
    scaled and rounded to bf16), made on the device as they are asked for"""

    def __init__(self, seed, std, small=()):
        self.seed, self.std, self.small = seed, std, dict(small)

    def normal(self, name, index, std=None):
        h = 0xCBF29CE484222325
        for b in name.encode():
            h = ((h ^ b) * 0x100000001B3) & M64
        z = (index + 1) * _signed(GOLDEN) + _signed(_mix(((self.seed * GOLDEN) & M64) ^ h))
        z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * _signed(0xBF58476D1CE4E5B9)
        z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * _signed(0x94D049BB133111EB)
        z = z ^ ((z >> 31) & ((1 << 33) - 1))
        s = (z & 0xFFFF) + ((z >> 16) & 0xFFFF) + ((z >> 32) & 0xFFFF) + ((z >> 48) & 0xFFFF)
        unit, std = (torch.tensor(v, dtype=torch.float32, device="cuda") for v in (1.0 / 37837.22719439421, self.std if std is None else std))
        return ((s - 131070).float() * unit * std).bfloat16().to(F64)

    def __call__(self, name, *shape):
        if name in self.small:
            return torch.from_numpy(self.small[name]).cuda().to(F64).reshape(shape)
        n = math.prod(shape)
        return torch.cat([self.normal(name, torch.arange(a, min(n, a + (1 << 26)), device="cuda")) for a in range(0, n, 1 << 26)]).reshape(shape)

    def rows(self, name, ids, width, std=None):
        ids = torch.as_tensor(np.asarray(ids).astype(np.int64), device="cuda")
        return self.normal(name, ids[:, None] * width + torch.arange(width, device="cuda"), std)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _swish_clamp(g, u, limit):
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


_silu = torch.nn.functional.silu


def _turn(x, pos, rot, halves):
    """rotary embedding of x [T, heads, channels] at positions pos: the leading rot["dims"] channels, YaRN where the entry says so"""
    n, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    i = torch.arange(n // 2, dtype=F64, device=x.device)
    f, mult = base ** (-2.0 * i / n), 1.0
    if sc:
        index = lambda turns: n * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(index(sc["fast"])), 0), min(math.ceil(index(sc["slow"])), n - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, mult = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    a = pos.to(F64)[:, None] * f
    c, s = (torch.cos(a) * mult)[:, None], (torch.sin(a) * mult)[:, None]
    y = x.clone()
    if halves:
        u, v = x[..., :n // 2], x[..., n // 2:n]
        y[..., :n // 2], y[..., n // 2:n] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., 0:n:2], x[..., 1:n:2]
        y[..., 0:n:2], y[..., 1:n:2] = u * c - v * s, v * c + u * s
    return y


def _attend(q, k, v, scale, window=0, keep_first=0, cap=0.0, sink=None, q_pos=None):
    """q [Tq, H, D] at positions q_pos, k / v [T, G, D | Dv]; sink: a score per head that joins the denominator -> [Tq, H Dv]"""
    H, rep = q.shape[1], q.shape[1] // k.shape[1]
    i = torch.arange(q.shape[0], device=q.device) if q_pos is None else q_pos
    j = torch.arange(k.shape[0], device=q.device)
    seen = j[None] <= i[:, None]
    if window:
        seen &= (i[:, None] - j[None] < window) | (j[None] < keep_first)
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h // rep].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
        out.append(torch.softmax(s, -1)[:, :k.shape[0]] @ v[:, h // rep])
    return torch.cat(out, -1)


def _recur(q, k, v, decay, beta=None):
    """S <- decay S + k v^T (with beta: the delta rule's corrected v), o = S^T q, token by token; q, k, decay [T, H, D | 1], v [T, H, Dv]"""
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * decay[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return out


def _experts(h, chosen, weight, one):
    """sum of weight x one(e, rows) over each row's chosen experts"""
    y = torch.zeros_like(h)
    for e in range(EXPERTS):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            y[rows] += weight[rows, place][:, None] * one(e, h[rows])
    return y


def _llama_exact(case, seed):
    _, H, I, V, heads, kv, eps, theta = LLAMA_FAMILY[case["model"]]
    d, w, qwen = H // heads, _Weights(seed, _std(H)), case["model"] == "qwen25_7b"
    decode = case["work"] == "decode"
    prefix, nxt = _llama_decode_tokens(case, seed) if decode else (_tokens(seed + 1, case["tokens"], V), [])
    n = len(prefix)
    lengths = torch.tensor(_lengths(case) if decode else [], device="cuda", dtype=torch.int64)
    # the shared prefix and, behind it, the new token of every sequence; a new token sees the part of the prefix its sequence holds and itself
    pos = torch.cat([torch.arange(n, device="cuda"), lengths])
    x = w.rows("model.embed_tokens.weight", np.concatenate([prefix, nxt]), H)
    rot = {"dims": d, "base": theta}
    for li in range(case["layers"]):
        p = f"model.layers.{li}."
        h = _rms(x, eps)

        def proj(m, rows):
            y = h @ w(f"{p}self_attn.{m}_proj.weight", rows, H).T
            return (y + w(f"{p}self_attn.{m}_proj.bias", rows) if qwen else y).reshape(-1, rows // d, d)
        q, k, v = _turn(proj("q", H), pos, rot, True), _turn(proj("k", kv * d), pos, rot, True), proj("v", kv * d)
        a = _attend(q[:n], k[:n], v[:n], d ** -0.5)
        if decode:
            own = [_attend(q[n + b:n + b + 1], torch.cat([k[:m], k[n + b:n + b + 1]]), torch.cat([v[:m], v[n + b:n + b + 1]]), d ** -0.5,
                           q_pos=torch.tensor([m], device="cuda")) for b, m in enumerate(lengths.tolist())]
            a = torch.cat([a] + own)
        x = x + a @ w(p + "self_attn.o_proj.weight", H, H).T
        h = _rms(x, eps)
        if case["model"] == "mixtral8x7b":
            e_ = p + "block_sparse_moe."
            s = torch.softmax(h @ w(e_ + "gate.weight", EXPERTS, H).T, -1)
            top, chosen = torch.topk(s, TOP)
            x = x + _experts(h, chosen, top / top.sum(-1, keepdim=True), lambda e, r: (
                _silu(r @ w(f"{e_}experts.{e}.w1.weight", I, H).T) * (r @ w(f"{e_}experts.{e}.w3.weight", I, H).T)) @ w(f"{e_}experts.{e}.w2.weight", H, I).T)
        else:
            x = x + (_silu(h @ w(p + "mlp.gate_proj.weight", I, H).T) * (h @ w(p + "mlp.up_proj.weight", I, H).T)) @ w(p + "mlp.down_proj.weight", H, I).T
    return _rms(x[n:] if decode else x[-1:], eps) @ w("lm_head.weight", V, H).T


def _embed_exact(case, seed):
    H, I, V, heads, b, t = 384, 1536, 30522, 12, case["batch"], case["tokens"]
    w, d = _Weights(seed, 0.02), H // heads
    ids = _tokens(seed + 1, b * t, V)

    def norm(x, name):
        m = x.mean(-1, keepdim=True)
        return (x - m) / torch.sqrt(((x - m) ** 2).mean(-1, keepdim=True) + 1e-12) + w(name + ".bias", H)

    def lin(x, name, rows, cols):
        return x @ w(name + ".weight", rows, cols).T + w(name + ".bias", rows)
    x = w.rows("embeddings.word_embeddings.weight", ids, H).reshape(b, t, H) + w("embeddings.position_embeddings.weight", 512, H)[:t]
    x = norm(x, "embeddings.LayerNorm")
    for i in range(6):
        p = f"encoder.layer.{i}."
        q, k, v = (lin(x, f"{p}attention.self.{n}", H, H).reshape(b, t, heads, d).transpose(1, 2) for n in ("query", "key", "value"))
        a = torch.softmax(q @ k.transpose(2, 3) / math.sqrt(d), -1) @ v
        x = norm(x + lin(a.transpose(1, 2).reshape(b, t, H), p + "attention.output.dense", H, H), p + "attention.output.LayerNorm")
        x = norm(x + lin(_gelu(lin(x, p + "intermediate.dense", I, H)), p + "output.dense", H, I), p + "output.LayerNorm")
    y = x.sum(1)
    return y / torch.sqrt((y * y).sum(-1, keepdim=True))


class _Layered:
    """one sequence of a layered model from its first token on; returns the logits of its last token"""

    def __init__(self, family, width, seed):
        self.family, self.W, self.cfg = family, width, _layered_config(family, width)
        self.w = _Weights(seed, _std(width), _small_tensors(self.cfg, family, seed))
        self.kept = {}

    def mat(self, name, *shape):
        """a matrix, kept for the sequences that follow as the bf16 values it holds"""
        if name not in self.kept:
            self.kept[name] = self.w(name, *shape).bfloat16()
        return self.kept[name].to(F64)

    def lin(self, x, name, rows):
        return x @ self.mat(name, rows, x.shape[-1]).T

    def softmax_attention(self, p, m, h, pos):
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k = self.lin(h, p + "q", H * D), self.lin(h, p + "k", G * D)

        def split(z, n):
            return z.reshape(-1, n, D)
        if self.family == "tufazen":
            q, k = split(q, H), split(k, G)
            o = _attend(_turn(q, pos, m["rot"], False), _turn(k, pos, m["rot"], False), k, m["scale"], cap=m["softcap"], sink=self.w(p + "sink", H))
            return self.lin(o * torch.sigmoid(self.lin(h, p + "g", H * D)), p + "o", self.W)
        v, whole = split(self.lin(h, p + "v", G * D), G), p.endswith("left.")
        q, k = (split(_rms(q, 1e-6), H), split(_rms(k, 1e-6), G)) if whole else (_rms(split(q, H), 1e-6), _rms(split(k, G), 1e-6))
        q, k = _turn(q, pos, m["rot"], True), _turn(k, pos, m["rot"], True)
        mask = m.get("mask") or {}
        o = _attend(q, k, v, m["scale"], window=mask["size"] if whole else 0, keep_first=mask.get("keep_first", 0), cap=m.get("softcap", 0.0),
                    sink=self.w(p + "sink", H) if whole else torch.zeros(H, dtype=F64, device="cuda"))
        return self.lin(o, p + "o", self.W)

    def latent_attention(self, p, m, h, pos):
        H, D, R, Dv, C, Q = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m.get("q_rank", 0)
        q = self.lin(_rms(self.lin(h, p + "dq", Q), 1e-6), p + "uq", H * (D + R)) if Q else self.lin(h, p + "q", H * (D + R))
        q, c = q.reshape(-1, H, D + R), self.lin(h, p + "dkv", C + R)
        # the fill lays a turned part's rows out as neighbouring pairs, whichever way the design pairs them
        kr = _turn(c[:, None, C:], pos, m["rot"], False).expand(-1, H, -1)
        lat = _rms(c[:, :C], 1e-6)
        k = torch.cat([torch.einsum("tc,hcd->thd", lat, self.mat(p + "uk", H, C, D)), kr], -1)
        v = torch.einsum("tc,hvc->thv", lat, self.mat(p + "uv", H, Dv, C))
        o = _attend(torch.cat([q[..., :D], _turn(q[..., D:], pos, m["rot"], False)], -1), k, v, m["scale"], window=(m.get("mask") or {}).get("size", 0))
        if self.family == "tufazen":
            o = (o.reshape(-1, H, Dv) * torch.sigmoid(self.lin(h, p + "g", H))[..., None]).reshape(-1, H * Dv)
        return self.lin(o, p + "o", self.W)

    def gla(self, p, m, h):
        H, D, Dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (self.lin(h, p + n, H * d).reshape(-1, H, d) for n, d in (("q", D), ("k", D), ("v", Dv)))
        z = self.lin(self.lin(h, p + "a1", 16), p + "a2", H * D) + 3.0
        o = _rms(_recur(q * D ** -0.5, k, v, torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(-1, H, D)), 1e-6).reshape(-1, H * Dv)
        return self.lin(o * _silu(self.lin(h, p + "g", H * Dv)), p + "o", self.W)

    def lightning(self, p, m, h):
        H, D, Dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(self.lin(h, p + n, H * d)).reshape(-1, H, d) for n, d in (("q", D), ("k", D), ("v", Dv)))
        decay = torch.tensor(np.float32(m["decay"]), device="cuda").to(F64).reshape(1, H, 1).expand(len(h), H, 1)
        o = _rms(_recur(q, k, v, decay).reshape(-1, H * Dv), 1e-6)
        return self.lin(o * torch.sigmoid(self.lin(h, p + "g", H * Dv)), p + "o", self.W)

    def conv(self, x, name):
        c = self.w(name, x.shape[1], 4)
        full = torch.cat([torch.zeros(3, x.shape[1], dtype=F64, device="cuda"), x])
        return sum(full[j:j + len(x)] * c[:, j] for j in range(4))

    def delta(self, p, m, h):
        H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(self.conv(self.lin(h, p + n, r), p + n + ".conv")) for n, r in (("q", G * D), ("k", G * D), ("v", H * Dv)))

        def unit(z):
            z = z.reshape(-1, G, D)
            return (z / torch.sqrt((z ** 2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
        decay = torch.exp(-torch.exp(self.w(p + "A_log", H)) * torch.nn.functional.softplus(self.lin(h, p + "a", H) + self.w(p + "dt_bias", H)))
        o = _rms(_recur(unit(q) * D ** -0.5, unit(k), v.reshape(-1, H, Dv), decay[..., None], torch.sigmoid(self.lin(h, p + "b", H))), 1e-6)
        return self.lin(o.reshape(-1, H * Dv) * _silu(self.lin(h, p + "g", H * Dv)), p + "o", self.W)

    def mamba2(self, p, m, h):
        H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * P
        z, xbc, dt = self.lin(h, p + "in", 2 * inner + 2 * G * N + H).split([inner, inner + 2 * G * N, H], -1)
        xbc = _silu(self.conv(xbc, p + "conv"))
        x, b, c = xbc.split([inner, G * N, G * N], -1)
        x, b, c = x.reshape(-1, H, P), b.reshape(-1, G, N).repeat_interleave(H // G, 1), c.reshape(-1, G, N).repeat_interleave(H // G, 1)
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias", H))
        y = _recur(c, b * dt[..., None], x, torch.exp(-torch.exp(self.w(p + "A_log", H)) * dt)[..., None]) + x
        return self.lin(_rms(y.reshape(-1, inner) * _silu(z), 1e-6), p + "o", self.W)

    def mixer(self, i, l, h, pos):
        p, m, kind = f"l{i}.mix.", l["mixer"], l["type"]
        if kind == "parallel":
            return 0.5 * self.softmax_attention(p + "left.", m["left"], h, pos) + 0.5 * self.lightning(p + "right.", m["right"], h)
        if kind in ("attention", "latent_attention"):
            return (self.softmax_attention if kind == "attention" else self.latent_attention)(p, m, h, pos)
        return getattr(self, kind)(p, m, h)

    def feed_forward(self, i, mlp, h):
        p, fam = f"l{i}.mlp.", self.family

        def glu(q, r, F):
            g, u = self.lin(r, q + "gate", F), self.lin(r, q + "up", F)
            a = _gelu(g) * u if fam == "rofetar" else _silu(g) * u if fam == "tufazen" and mlp["kind"] == "moe" else _swish_clamp(g, u, 7.0)
            return self.lin(a, q + "down", self.W)
        if mlp["kind"] == "dense":
            return glu(p, h, mlp["ff"])
        s = self.lin(h, p + "router", EXPERTS)
        s = torch.softmax(s + self.w(p + "router.b", EXPERTS) if fam == "medulorn" else s, -1)
        if fam == "tufazen":
            groups = mlp["router"]["groups"]
            best = s.reshape(len(h), groups["count"], -1).amax(-1)
            keep = torch.zeros_like(best).scatter(1, torch.topk(best, groups["keep"]).indices, 1.0)
            top, chosen = torch.topk(s * keep.repeat_interleave(EXPERTS // groups["count"], 1), TOP)
        else:
            top, chosen = torch.topk(s, TOP)
            top = top / top.sum(-1, keepdim=True)
        shared = glu(p + "shared.", h, mlp["shared"]["ff"])
        if fam == "nifunex":
            shared = shared * torch.sigmoid(self.lin(h, p + "shared.sg", 1))
        return shared + _experts(h, chosen, top, lambda e, r: glu(f"{p}e{e}.", r, mlp["expert"]["ff"]))

    def __call__(self, ids):
        fam, W, w, cfg = self.family, self.W, self.w, self.cfg
        pos = torch.arange(len(ids), device="cuda")
        x = w.rows("embed", ids, W, 1.0)
        if fam == "tufazen":
            b = cfg["embedding"]["bigram"]
            prev = np.concatenate([[0], ids[:-1].astype(np.int64)])
            row = (prev * b["mul_prev"] + ids.astype(np.int64) * b["mul_cur"]) % b["buckets"]
            row[0] = b["buckets"]
            x = x + w.rows("bigram", row, W, 1.0)
        for i, l in enumerate(cfg["layers"]):
            if fam == "medulorn":
                before = torch.cat([torch.zeros(1, W, dtype=F64, device="cuda"), x[:-1]])
                x = _rms(x + self.mixer(i, l, x + (before - x) * w(f"l{i}.shift", W), pos), 1e-6)
                x = _rms(x + self.feed_forward(i, l["mlp"], x), 1e-6)
            elif fam == "tufazen":
                h = torch.tanh(0.5 * x)
                x = x + self.mixer(i, l, h, pos) + self.feed_forward(i, l["mlp"], h)
                S, n = cfg["token_side"]["dim"], len(cfg["layers"])
                e = w.rows("side.embed", ids, n * S, 1.0)[:, i * S:(i + 1) * S]
                x = x + _rms(self.lin(_gelu(self.lin(x, f"l{i}.side.gate", S)) * e, f"l{i}.side.proj", W), 1e-6)
            elif fam == "rofetar":
                x = x + _rms(self.mixer(i, l, x, pos), 1e-6)
                x = x + _rms(self.feed_forward(i, l["mlp"], x), 1e-6)
            else:
                x = x + _rms(self.mixer(i, l, _rms(x, 1e-6), pos), 1e-6)
                x = x + _rms(self.feed_forward(i, l["mlp"], _rms(x, 1e-6)), 1e-6)
        x = x[-1:]
        z = self.lin(torch.tanh(0.5 * x) if fam == "tufazen" else _rms(x, 1e-6), "head", LAYERED_VOCAB)
        return 50.0 * torch.tanh(z / 50.0) if fam == "medulorn" else z


def exact(case, seed):
    with torch.no_grad():
        if case["work"] == "embed":
            return _embed_exact(case, seed)
        if case["work"] != "step":
            return _llama_exact(case, seed)
        held, nxt, portion = _step_tokens(case, seed)
        model = _Layered(case["model"], case["width"], seed)
        sequences = [np.concatenate([h, [t]]) for h, t in zip(held, nxt)] + ([portion] if case["tokens"] else [])
        return torch.cat([model(s) for s in sequences])
