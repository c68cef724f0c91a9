"""Timed cases: the steps that a serving loop has the engine run, through its public Python interface.

A pass is one ``Engine.forward_batch`` and the wait for its tokens, which is what a scheduler does before it can build
the next batch: a decode step of a batch of running requests (captured as a CUDA graph, as a server captures them at its
start), or a prefill step of a few prompts, in whole or behind a cached prefix.  Models are the ones this repository's
benchmark runs: Qwen3-0.6B, Llama-3-8B, a Qwen3-MoE model of 64 experts and a Saluzen layer stack (attention beside
recurrences, latent attention).  Weights, caches and prompts are drawn from the seed; lengths belong to the case.

The drawn weights keep two properties of trained ones without which outputs could not be compared: the next token stands
out (the output head knows the embedding), and so do a token's experts (some columns of the residual carry them).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()
from sglang_cpp_b200 import models, weights  # noqa: E402
from sglang_cpp_b200.engine import Engine, EngineConfig  # noqa: E402

f64, bf16 = torch.float64, torch.bfloat16
PREFILL, DECODE = 0, 1
MAX_REQUESTS, MAX_LEN, MAX_EXTEND = 64, 8192, 8192   # what the engine is made for, whatever a case asks of it
PAGE = 16
LOGIT_GAIN = 0.08                                    # final norm: logits spread over a few units


def _dense(layers, width, q_heads, kv_heads, ff, vocab, theta, tied, qk_norm, experts=0, top=0):
    return models.ModelConfig(layers, width, q_heads, kv_heads, 128, ff, vocab, 1e-6, theta, MAX_LEN, tied, qk_norm, qk_norm,
                              "silu", experts, top, ff if experts else 0)


UNIFORM = {
    "qwen3-0.6b": _dense(28, 1024, 16, 8, 3072, 151936, 1e6, True, True),
    "llama-3-8b": _dense(32, 4096, 32, 8, 14336, 128256, 5e5, False, False),
    "qwen3-moe": _dense(12, 2048, 16, 4, 1024, 32768, 1e6, False, True, 64, 4),
}


def _saluzen_config():
    """Six layers 2048 wide: attention in chunks beside the delta rule, latent attention (the second one on the latents of
    the first), attention beside the state space."""
    width, heads, kv_heads, ff = 2048, 16, 4, 6144
    attention = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    scaling = {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192.0}
    layers = []
    for i in range(6):
        if i % 3 == 0:
            left = {**attention, "rot": {"base": 1e6, "dims": 128}, "mask": {"size": 1536}}
            m = {"left": left, "left_scale": 0.8, "right_scale": 1.0,
                 "right": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}}
            kind = "parallel_2"
        elif i % 3 == 1:
            m = {"heads": heads, "dim": 64, "rot_dim": 64, "vdim": 128, "q_rank": 768, "kv_rank": 512, "scale": 128 ** -0.5,
                 "rot": {"base": 1e4, "dims": 64}}
            if i == 4:
                m["kv_from"] = 1
            kind = "latent_attention"
        else:
            m = {"left": {**attention, "rot": {"base": 1e6, "dims": 128, "scaling": scaling}},
                 "right": {"heads": width // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}}
            kind = "parallel"
        layers.append({"type": kind, "mixer": m, "mlp": {"kind": "dense", "ff": ff}})
    return {"architecture": "Saluzen", "width": width, "vocab": 32768, "norm": {"eps": 1e-6}, "layers": layers}


SALUZEN = _saluzen_config()


# ---- cases -------------------------------------------------------------------------

def _case(model, step, requests, lo, hi, cached=0, sampled=False, lens=1):
    """``lo`` to ``hi``: tokens in the cache of every decoded request, or new tokens of every prompt behind ``cached``
    cached ones.  ``lens`` seeds the lengths."""
    return {"model": model, "step": step, "requests": requests, "lo": lo, "hi": hi, "cached": cached, "sampled": sampled, "lens": lens}


def listed():
    def named(name, *a, **k):
        return {"name": name, **_case(*a, **k)}
    return [
        # one user's chat: the smallest call, where latency is everything
        named("qwen3 decode 1", "qwen3-0.6b", "decode", 1, 700, 700),
        # a few users, sampling, a batch that fills no captured size
        named("qwen3 decode 5 sampled", "qwen3-0.6b", "decode", 5, 200, 3000, sampled=True),
        # a loaded server: the batch this repository's benchmark decodes
        named("qwen3 decode 64", "qwen3-0.6b", "decode", 64, 512, 2048),
        # time to the first token of a short question
        named("qwen3 prefill 1 short", "qwen3-0.6b", "prefill", 1, 181, 181),
        # a prefill batch as the scheduler forms them from ragged prompts
        named("qwen3 prefill 6", "qwen3-0.6b", "prefill", 6, 512, 2048),
        # long prompts advancing in chunks: new tokens behind a cached prefix
        named("qwen3 prefill 4 chunks", "qwen3-0.6b", "prefill", 4, 2048, 2048, cached=2048),
        # a larger dense model, few users: weights are read for every token
        named("llama decode 4", "llama-3-8b", "decode", 4, 500, 1500),
        # ... and a long document handed to it: the largest call
        named("llama prefill 2", "llama-3-8b", "prefill", 2, 1500, 2048),
        # mixture of experts, a server's batch and a prompt batch
        named("moe decode 32", "qwen3-moe", "decode", 32, 300, 2000),
        named("moe prefill 3", "qwen3-moe", "prefill", 3, 700, 1800),
        # recurrent and latent layers, decoding for a group of users, and one long prompt
        named("saluzen decode 16", "saluzen", "decode", 16, 200, 900),
        named("saluzen prefill 1", "saluzen", "prefill", 1, 3001, 3001),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["qwen3-0.6b", "qwen3-0.6b", "llama-3-8b", "qwen3-moe", "saluzen"])
    lens = rng.randrange(1, 1 << 20)
    if rng.random() < 0.55:
        top = {"saluzen": 900, "llama-3-8b": 2048}.get(model, 4000)
        requests = spread(1, 24 if model == "saluzen" else 64)
        hi = spread(100, top)
        return _case(model, "decode", requests, max(64, hi // 4), hi, sampled=rng.random() < 0.3, lens=lens)
    requests = rng.randint(1, 6)
    most = {"llama-3-8b": 3000, "saluzen": 4000}.get(model, 8000) // requests
    hi = spread(60, most)
    cached = PAGE * rng.randint(1, 128) if model != "saluzen" and rng.random() < 0.4 else 0
    return _case(model, "prefill", requests, max(33, hi // 3), hi, cached=cached, lens=lens)


def _lengths(case):
    """(cached tokens, new tokens) of every request."""
    rng = random.Random(case["lens"])
    n = [rng.randint(case["lo"], case["hi"]) for _ in range(case["requests"])]
    if case["step"] == "decode":
        return n, [1] * len(n)
    return [case["cached"]] * len(n), n


def _tokens(case, seed):
    """Token ids of every request, those in the cache included."""
    vocab = SALUZEN["vocab"] if case["model"] == "saluzen" else UNIFORM[case["model"]].vocab_size
    rng = np.random.default_rng(seed)
    return [rng.integers(0, vocab, size=c + n).astype(np.int32) for c, n in zip(*_lengths(case))]


# ---- drawn weights -----------------------------------------------------------------

def _generator(seed, *where):
    at = 0
    for w in where:
        at = at * 1009 + w
    return torch.Generator(device="cuda").manual_seed(seed * 1000003 + at)


def _fill_uniform(cfg, t, name, layer, seed):
    """Draws one tensor of a grouped-query model into ``t`` (bf16, of its shape)."""
    kinds = ("embed", "lm_head", "final_norm", "qkv", "o", "input_norm", "post_norm", "q_norm", "k_norm", "router",
             "experts_gate_up", "experts_down", "gate_up", "down")
    g = _generator(seed, kinds.index(name), layer)
    E = cfg.num_experts
    if name == "final_norm":
        return t.fill_(LOGIT_GAIN)
    if name in ("q_norm", "k_norm"):
        return t.fill_(1.25 if name == "q_norm" else 1.0)     # scores spread over a few units
    if name.endswith("norm"):
        t.normal_(1.0, 0.1, generator=g)
        if E:
            t[:E] = 1
        return t
    if name == "router":        # an expert reads its own column, another one in every layer
        t.zero_()
        t[torch.randperm(E, device="cuda", generator=g), torch.arange(E, device="cuda")] = 0.5
        return t
    gain = 0.4 if name in ("o", "down", "experts_down") else 1.0     # (a block moves the residual a little, as in a trained model)
    t.normal_(0.0, 1.0 if name in ("embed", "lm_head") else gain * t.shape[-1] ** -0.5, generator=g)
    if name == "embed" and E:   # the columns that routers read: a token's experts stand out, and nothing is added to them
        code = torch.rand(t.shape[0], E, device="cuda", generator=g) * 2 - 1
        chosen = torch.rand(t.shape[0], E, device="cuda", generator=g).topk(cfg.num_experts_per_tok, dim=1).indices
        code.scatter_(1, chosen, (3 - 0.4 * torch.arange(cfg.num_experts_per_tok, device="cuda")).expand(t.shape[0], -1))
        t[:, :E] = code.to(bf16)
    if name == "lm_head":
        e = _fill_uniform(cfg, torch.empty_like(t), "embed", 0, seed)
        t.mul_(0.8).add_(e, alpha=0.6)
    if name == "qkv" and not cfg.qk_norm:
        t[:cfg.num_qo_heads * 128].mul_(1.25)
    if E and name == "o":
        t[:E] = 0
    if E and name == "experts_down":
        t[:, :E] = 0
    return t


def _shapes(cfg):
    """name -> shape of the tensors of one layer (and, under None, of the model)."""
    H, q, kv = cfg.hidden_size, cfg.num_qo_heads * 128, cfg.num_kv_heads * 128
    layer = {"qkv": (q + 2 * kv, H), "o": (H, q), "input_norm": (H,), "post_norm": (H,)}
    if cfg.qk_norm:
        layer.update(q_norm=(128,), k_norm=(128,))
    if cfg.num_experts:
        E, I = cfg.num_experts, cfg.moe_intermediate_size
        layer.update(router=(E, H), experts_gate_up=(E, 2 * I, H), experts_down=(E, H, I))
    else:
        layer.update(gate_up=(2 * cfg.intermediate_size, H), down=(H, cfg.intermediate_size))
    model = {"embed": (cfg.vocab_size, H), "final_norm": (H,)}
    if not cfg.tie_word_embeddings:
        model["lm_head"] = (cfg.vocab_size, H)
    return layer, model


def _saluzen_weights(seed):
    """Tensors of the Saluzen model by their names in a checkpoint."""
    w, D, V = {}, SALUZEN["width"], SALUZEN["vocab"]
    g = _generator(seed, 77)

    def normal(*shape, mean=0.0, std=1.0):
        return torch.empty(*shape, device="cuda").normal_(mean, std, generator=g).to(bf16)

    def mat(name, n, k, gain=1.0):
        w[name] = normal(n, k, std=gain * k ** -0.5)

    def vec(name, n, mean=1.0, std=0.1):
        w[name] = normal(n, mean=mean, std=std)

    def uniform(name, n, lo, hi):
        w[name] = (torch.rand(n, device="cuda", generator=g) * (hi - lo) + lo).to(bf16)

    def attention(p, m, gates):
        for t, n, gain in (("q", m["heads"] * m["dim"], 1.4), ("k", m["kv_heads"] * m["dim"], 1.4), ("v", m["kv_heads"] * m["vdim"], 1.0)):
            mat(p + t, n, D, gain)
            vec(f"{p}{t}.b", n, 0.0, 0.2)
        mat(p + "g", gates, D)
        mat(p + "o", D, m["heads"] * m["vdim"])

    w["embed"] = normal(V, D, std=2.0)
    for i, layer in enumerate(SALUZEN["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        for norm in ("norm1", "norm1b", "norm2", "norm2b"):
            vec(p + norm, D)
        if layer["type"] == "latent_attention":
            H, d, dr, dv, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            mat(p + "mix.dq", m["q_rank"], D)
            vec(p + "mix.dq.norm", m["q_rank"])
            mat(p + "mix.uq", H * (d + dr), m["q_rank"], 1.4)
            if m.get("kv_from") is None:
                mat(p + "mix.dkv", r + dr, D)
                vec(p + "mix.dkv.norm", r)
            mat(p + "mix.uk", H * d, r, 1.4)
            mat(p + "mix.uv", H * dv, r)
            mat(p + "mix.o", D, H * dv)
        else:
            left, right, r = p + "mix.left.", p + "mix.right.", m["right"]
            H, dv = r["heads"], r["vdim"]
            if layer["type"] == "parallel":
                attention(left, m["left"], m["left"]["heads"] * m["left"]["vdim"])
                inner, gn = H * dv, r["groups"] * r["state"]
                mat(right + "in", 2 * inner + 2 * gn + H, D)
                w[right + "conv"] = normal(inner + 2 * gn, r["conv"], std=0.6)
                vec(right + "conv.b", inner + 2 * gn, 0.0, 0.2)
                vec(right + "D", H, 0.5, 0.3)
                vec(right + "norm", inner)
                vec(p + "mix.left.out", D)
                vec(p + "mix.right.out", D)
            else:
                attention(left, m["left"], m["left"]["heads"])
                vec(left + "sink", m["left"]["heads"], 0.5, 1.0)
                G, d = r["kv_heads"], r["dim"]
                for t, n in (("q", G * d), ("k", G * d), ("v", H * dv)):
                    mat(right + t, n, D)
                    w[f"{right}{t}.conv"] = normal(n, r["conv"], std=0.6)
                mat(right + "a", H, D)
                mat(right + "b", H, D)
                mat(right + "g", H * dv, D)
                vec(right + "norm", dv)
            uniform(right + "A_log", H, -2.0, 1.0)
            uniform(right + "dt_bias", H, -5.0, -1.0)
            mat(right + "o", D, H * dv)
        ff = layer["mlp"]["ff"]
        mat(p + "mlp.gate", ff, D)
        mat(p + "mlp.up", ff, D)
        mat(p + "mlp.down", D, ff)
    w["final.norm"] = torch.full((D,), LOGIT_GAIN, device="cuda", dtype=bf16)
    w["head"] = (0.3 * w["embed"].float() + 0.8 * normal(V, D).float()).to(bf16)
    return w


# ---- what a server has in hand before a step -----------------------------------------

def _pages(case, seed):
    """Pages of every request, and how many of the first pages the step writes into: a pool that has been in use hands its
    pages out in no order.  (Those that the step writes come first, so that they can be returned by themselves.)"""
    cached, new = _lengths(case)
    held = [-(-(c + n) // PAGE) for c, n in zip(cached, new)]
    before = [c // PAGE for c in cached]
    written = sum(h - b for h, b in zip(held, before))
    rng = np.random.default_rng(seed + 1)
    fresh = iter(rng.permutation(written).tolist())
    old = iter((written + rng.permutation(sum(before))).tolist())
    return [[next(old) for _ in range(b)] + [next(fresh) for _ in range(h - b)] for h, b in zip(held, before)], written


def _slots(pages, n):
    """The slots of a request's first n positions."""
    at = np.arange(n)
    return np.asarray(pages, dtype=np.int64)[at // PAGE] * PAGE + at % PAGE


def _draw_cache(cfg, cache, written, case, seed):
    """Keys and values of cached tokens; places that the step writes and nothing is cached in are zero."""
    cache.normal_(0.0, 1.0, generator=_generator(seed, 91))
    if case["step"] == "prefill":
        cache[:, :, :written * PAGE] = 0


class _Owned:
    """An engine's tensor, as an object that torch can view and that keeps the engine: a view may outlive its state."""

    def __init__(self, engine, name, layer):
        self.engine = engine
        at, nbytes = engine.tensor_info(name, layer)
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (at, False), "version": 3, "strides": None}


def _view(engine, name, layer=0, dtype=bf16):
    return torch.as_tensor(_Owned(engine, name, layer), device="cuda").view(dtype)


def prepare(case, seed):
    cached, new = _lengths(case)
    rows = np.arange(case["requests"], dtype=np.int32)
    pages, written = _pages(case, seed)
    tokens = _tokens(case, seed)
    stack = case["model"] == "saluzen"
    cfg = models.read_saluzen(SALUZEN) if stack else UNIFORM[case["model"]]
    e = Engine(cfg, EngineConfig(PAGE, sum(map(len, pages)) + 1, MAX_REQUESTS, MAX_LEN, MAX_EXTEND))
    out = {}
    if stack:
        e.load_weights(weights.pack_layer_stack(cfg, {k: t.cpu() for k, t in _saluzen_weights(seed).items()}))
    else:
        layer, model = _shapes(cfg)
        for l in range(cfg.num_layers):
            for name, shape in layer.items():
                _fill_uniform(cfg, _view(e, name, l).view(shape), name, l, seed)
        for name, shape in model.items():
            _fill_uniform(cfg, _view(e, name).view(shape), name, 0, seed)
        cache = _view(e, "kv_cache").view(2, cfg.num_layers, -1, cfg.num_kv_heads, 128)
        _draw_cache(cfg, cache, written, case, seed)
        out["cache"] = cache[:, :, :written * PAGE]
    torch.cuda.synchronize()
    for r, p, t in zip(rows, pages, tokens):
        at = np.arange(len(t), dtype=np.int32)
        e.write_page_table(np.full(len(t), r, np.int32), at, _slots(p, len(t)).astype(np.int32))
        e.write_token_pool(np.full(len(t), r, np.int32), at, t)
    if stack and case["step"] == "decode":   # a state is what the prompt leaves behind
        for i in range(0, len(rows), 8):
            part = slice(i, i + 8)
            e.forward_batch(PREFILL, rows[part], np.zeros(len(rows[part]), np.int32), cached[part],
                            write_pos=[-1] * len(rows[part])).synchronize()
    if stack:
        for i, entry in enumerate(SALUZEN["layers"]):
            if entry["type"] != "latent_attention":
                r = entry["mixer"]["right"]
                shape = (-1, r["heads"], r.get("state") or r["dim"], r["vdim"])
                out[f"state{i}"] = _view(e, "beside_state", i, torch.float32).view(shape)[:len(rows)]
    if case["step"] == "decode":
        e.capture_graphs([1 << (len(rows) - 1).bit_length()])
    vocab = cfg.vocab_size
    out["logits"] = _view(e, "logits").view(-1, vocab)[:len(rows)]
    step = dict(phase=DECODE if case["step"] == "decode" else PREFILL, table_idx=rows, cached_lens=np.asarray(cached, np.int32),
                extend_lens=np.asarray(new, np.int32), write_pos=np.asarray([c + n for c, n in zip(cached, new)], np.int32))
    if case["sampled"]:
        step.update(temperatures=np.full(len(rows), 0.7, np.float32), top_k=np.full(len(rows), 50, np.int32),
                    top_p=np.full(len(rows), 0.9, np.float32), seeds=np.arange(len(rows), dtype=np.uint64) + seed)
    torch.cuda.synchronize()
    return {"engine": e, "step": step, "out": out}


def run(state):
    done = state["engine"].forward_batch(**state["step"])
    done.synchronize()
    return {"tokens": done.next_tokens_cpu, **state["out"]}


# ---- what a step cannot do without ---------------------------------------------------

def _pairs(case):
    """(query, key) pairs of causal attention."""
    return sum(n * c + n * (n + 1) / 2 for c, n in zip(*_lengths(case)))


def work(case):
    cached, new = _lengths(case)
    B, T, keys = len(new), sum(new), sum(cached) + sum(new)
    if case["model"] != "saluzen":
        cfg = UNIFORM[case["model"]]
        H, q, kv, L, V = cfg.hidden_size, cfg.num_qo_heads * 128, cfg.num_kv_heads * 128, cfg.num_layers, cfg.vocab_size
        attn = H * (q + 2 * kv) + q * H
        expert = 3 * H * (cfg.moe_intermediate_size or cfg.intermediate_size)
        used, read = expert, expert
        if cfg.num_experts:
            E, top = cfg.num_experts, cfg.num_experts_per_tok
            used, read = top * expert, E * (1 - (1 - top / E) ** T) * expert + E * H
        return {"bytes": 2 * (L * (attn + read) + V * H) + 4 * L * kv * keys + 2 * T * H + 2 * B * V,
                "flops": 2 * T * L * (attn + used) + 2 * B * V * H + 4 * L * q * _pairs(case)}
    D, V = SALUZEN["width"], SALUZEN["vocab"]
    size = flops = state = 0
    cache = 0.0
    for i, layer in enumerate(SALUZEN["layers"]):
        m = layer["mixer"]
        size += 3 * D * layer["mlp"]["ff"]
        if layer["type"] == "latent_attention":
            H, d, r = m["heads"], m["dim"] + m["rot_dim"], m["kv_rank"] + m["rot_dim"]
            size += D * m["q_rank"] + H * d * m["q_rank"] + H * (m["dim"] + m["vdim"]) * m["kv_rank"] + H * m["vdim"] * D
            size += D * r if m.get("kv_from") is None else 0
            cache += 2 * keys * r
            flops += 2 * H * (d + m["vdim"]) * _pairs(case)
            continue
        a, r = m["left"], m["right"]
        inner, n = r["heads"] * r["vdim"], r.get("state") or r["dim"]
        size += 2 * D * (a["heads"] + a["kv_heads"]) * 128 + 2 * D * inner + 2 * D * (r.get("groups") or r["kv_heads"]) * n
        size += D * inner + D * (a["heads"] * 128 if layer["type"] == "parallel" else a["heads"])
        chunk = (a.get("mask") or {}).get("size", MAX_LEN)
        pairs = sum(sum(p % chunk + 1 for p in range(c, c + t)) for c, t in zip(cached, new))
        seen = sum((c + t - 1) % chunk + 1 if t == 1 else c + t for c, t in zip(cached, new))
        cache += 2 * 2 * a["kv_heads"] * 128 * seen
        flops += 4 * a["heads"] * 128 * pairs + 4 * T * inner * n
        state += 4 * B * inner * n * (2 if case["step"] == "decode" else 1)
    return {"bytes": 2 * (size + V * D) + cache + state + 2 * T * D + 2 * B * V, "flops": flops + 2 * T * size + 2 * B * V * D}


def tolerance(case):
    """bf16 activations and a bf16 residual stream through all layers.  Measured with the norms and head operations folded
    into the projections against the kernels apart from them, two correct orders of the same sums: logits rel 0.018,
    max 0.1, which is what either is from 64 bits as well (28 layers round the residual 56 times); no token differs."""
    return {"rel": 0.03, "max": 0.5, "differ": 0.0}


# ---- the same in 64 bits -------------------------------------------------------------

def _norm(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, angles, neighbours=False):
    """Rotates the first 2 * angles.shape[1] elements of x [n, heads, d]; the pairs are halves, or neighbours."""
    h = angles.shape[1]
    c, s = torch.cos(angles)[:, None], torch.sin(angles)[:, None]
    u, v = (x[..., 0:2 * h:2], x[..., 1:2 * h:2]) if neighbours else (x[..., :h], x[..., h:2 * h])
    y = (u * c - v * s, v * c + u * s)
    return torch.cat([torch.stack(y, -1).flatten(-2) if neighbours else torch.cat(y, -1), x[..., 2 * h:]], -1)


def _frequencies(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, device="cuda", dtype=f64) / dims)


def _attend(q, k, v, scale, first, chunk=None, sink=None):
    """q [n, Hq, d] at positions first.. over k, v [m, Hkv, d] at positions 0.. (causal; within chunks; with a sink)."""
    n, H, m = q.shape[0], q.shape[1], k.shape[0]
    i, j = first + torch.arange(n, device="cuda")[:, None], torch.arange(m, device="cuda")[None]
    hidden = j > i if chunk is None else (j > i) | (i // chunk != j // chunk)
    out = torch.empty(n, H, v.shape[2], device="cuda", dtype=f64)
    per = H // k.shape[1]
    for h in range(H):
        s = (q[:, h] @ k[:, h // per].T * scale).masked_fill_(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :m] @ v[:, h // per]
    return out


def _exact_uniform(case, seed):
    cfg = UNIFORM[case["model"]]
    cached, new = _lengths(case)
    pages, written = _pages(case, seed)
    Hq, Hk, eps = cfg.num_qo_heads, cfg.num_kv_heads, cfg.rms_norm_eps
    layer, model = _shapes(cfg)

    def weight(name, l=0):
        return _fill_uniform(cfg, torch.empty((layer if name in layer else model)[name], device="cuda", dtype=bf16), name, l, seed).to(f64)

    tokens = torch.cat([torch.from_numpy(t[c:]).cuda().long() for t, c in zip(_tokens(case, seed), cached)])
    embed = _fill_uniform(cfg, torch.empty(model["embed"], device="cuda", dtype=bf16), "embed", 0, seed)
    x = embed[tokens].to(f64)
    del embed
    slots = (sum(map(len, pages)) + 2) * PAGE
    cache = torch.empty(2, cfg.num_layers, slots, Hk, 128, device="cuda", dtype=bf16)
    _draw_cache(cfg, cache, written, case, seed)
    fresh = cache[:, :, :written * PAGE].to(f64)
    where = [torch.from_numpy(_slots(p, c + n)).cuda() for p, c, n in zip(pages, cached, new)]
    angles = [torch.arange(c, c + n, device="cuda", dtype=f64)[:, None] * _frequencies(128, cfg.rope_theta) for c, n in zip(cached, new)]
    for l in range(cfg.num_layers):
        h = _norm(x, weight("input_norm", l), eps)
        q, k, v = (h @ weight("qkv", l).T).view(len(x), -1, 128).split([Hq, Hk, Hk], 1)
        if cfg.qk_norm:
            q, k = _norm(q, weight("q_norm", l), eps), _norm(k, weight("k_norm", l), eps)
        out, at = [], 0
        for b, (c, n) in enumerate(zip(cached, new)):
            mine, at = slice(at, at + n), at + n
            kb, vb = _turn(k[mine], angles[b]), v[mine]
            fresh[0, l, where[b][c:]], fresh[1, l, where[b][c:]] = kb, vb
            old = where[b][:c]
            out.append(_attend(_turn(q[mine], angles[b]), torch.cat([cache[0, l, old].to(f64), kb]),
                               torch.cat([cache[1, l, old].to(f64), vb]), 128 ** -0.5, c))
        x = x + torch.cat(out).flatten(1) @ weight("o", l).T
        h = _norm(x, weight("post_norm", l), eps)
        if not cfg.num_experts:
            gate, up = (h @ weight("gate_up", l).T).chunk(2, 1)
            x = x + (torch.nn.functional.silu(gate) * up) @ weight("down", l).T
            continue
        top = torch.softmax(h @ weight("router", l).T, 1).topk(cfg.num_experts_per_tok, 1)
        share = top.values / top.values.sum(1, keepdim=True)
        gate_up, down = weight("experts_gate_up", l), weight("experts_down", l)
        y = torch.zeros_like(x)
        for e in range(cfg.num_experts):
            t, place = torch.nonzero(top.indices == e, as_tuple=True)
            gate, up = (h[t] @ gate_up[e].T).chunk(2, 1)
            y.index_add_(0, t, share[t, place][:, None] * ((torch.nn.functional.silu(gate) * up) @ down[e].T))
        x = x + y
    last = torch.cumsum(torch.tensor(new, device="cuda"), 0) - 1
    head = weight("embed" if cfg.tie_word_embeddings else "lm_head")
    return {"tokens": None, "logits": _norm(x[last], weight("final_norm"), eps) @ head.T, "cache": fresh}


def _scaled_frequencies(rot):
    f, sc = _frequencies(rot["dims"], rot["base"]), rot.get("scaling")
    if not sc:
        return f
    wave = 2 * math.pi / f
    mix = ((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
    return (1 - mix) * f / sc["factor"] + mix * f


def _grouped(h, w, p, m, sink):
    n = len(h)
    q, k, v = ((h @ w[p + t].T + w[f"{p}{t}.b"]).view(n, -1, 128) for t in "qkv")
    angles = torch.arange(n, device="cuda", dtype=f64)[:, None] * _scaled_frequencies(m["rot"])
    o = _attend(_turn(q, angles), _turn(k, angles), v, m["scale"], 0, (m.get("mask") or {}).get("size"), sink)
    gate = torch.sigmoid(h @ w[p + "g"].T)
    return (o * gate.view(n, m["heads"], -1)).flatten(1) @ w[p + "o"].T


def _convolve(x, taps, bias=0.0):
    T = taps.shape[1]
    padded = torch.cat([x.new_zeros(T - 1, x.shape[1]), x])
    return torch.nn.functional.silu(sum(padded[i:i + len(x)] * taps[:, i] for i in range(T)) + bias)


def _latent(h, w, p, m, eps, kept):
    n, H, d, dr, r = len(h), m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    angles = torch.arange(n, device="cuda", dtype=f64)[:, None] * _frequencies(dr, m["rot"]["base"])
    q = (_norm(h @ w[p + "dq"].T, w[p + "dq.norm"], eps) @ w[p + "uq"].T).view(n, H, d + dr)
    q = torch.cat([_turn(q[..., d:], angles, True), q[..., :d]], -1)
    if m.get("kv_from") is None:
        z = h @ w[p + "dkv"].T
        kept["latent"] = _norm(z[:, :r], w[p + "dkv.norm"], eps), _turn(z[:, None, r:], angles, True)
    c, turned = kept["latent"]
    k = torch.cat([turned.expand(n, H, dr), (c @ w[p + "uk"].T).view(n, H, d)], -1)
    return _attend(q, k, (c @ w[p + "uv"].T).view(n, H, -1), m["scale"], 0).flatten(1) @ w[p + "o"].T


def _state_space(h, w, p, m, eps):
    n, H, dv, N, G = len(h), m["heads"], m["vdim"], m["state"], m["groups"]
    z, xbc, dt = (h @ w[p + "in"].T).split([H * dv, H * dv + 2 * G * N, H], 1)
    x, B, C = _convolve(xbc, w[p + "conv"], w[p + "conv.b"]).split([H * dv, G * N, G * N], 1)
    x = x.reshape(n, H, dv)
    B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"], threshold=1e9)
    decay, y = torch.exp(-torch.exp(w[p + "A_log"]) * dt), torch.empty_like(x)
    S = x.new_zeros(H, N, dv)
    for t in range(n):
        S.mul_(decay[t, :, None, None]).baddbmm_(B[t, :, :, None], (dt[t, :, None] * x[t])[:, None])
        y[t] = torch.bmm(C[t, :, None], S)[:, 0]
    y = (y + w[p + "D"][:, None] * x).flatten(1) * torch.nn.functional.silu(z)
    return (_norm(y.view(n, m["norm_groups"], -1), 1.0, eps).flatten(1) * w[p + "norm"]) @ w[p + "o"].T, S


def _delta_rule(h, w, p, m, eps):
    n, H, G, d, dv = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_convolve(h @ w[p + t].T, w[f"{p}{t}.conv"]) for t in "qkv")
    q, k = (t.view(n, G, d).repeat_interleave(H // G, 1) for t in (q, k))
    q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, v, y = q * d ** -0.5, v.view(n, H, dv), h.new_empty(n, H, dv)
    beta = torch.sigmoid(h @ w[p + "b"].T)
    step = torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"], threshold=1e9)
    decay = torch.exp(-torch.exp(w[p + "A_log"]) * step)
    S = h.new_zeros(H, d, dv)
    for t in range(n):
        S.mul_(decay[t, :, None, None])
        u = beta[t, :, None, None] * (v[t][:, None] - torch.bmm(k[t, :, None], S))
        S.baddbmm_(k[t, :, :, None], u)
        y[t] = torch.bmm(q[t, :, None], S)[:, 0]
    y = _norm(y, w[p + "norm"], eps).flatten(1)
    return (y * torch.nn.functional.silu(h @ w[p + "g"].T)) @ w[p + "o"].T, S


def _exact_saluzen(case, seed):
    w = {k: t.to(f64) for k, t in _saluzen_weights(seed).items()}
    eps, logits, states = SALUZEN["norm"]["eps"], [], {}
    for tokens in _tokens(case, seed):
        x, kept = w["embed"][torch.from_numpy(tokens).cuda().long()], {}
        for i, layer in enumerate(SALUZEN["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = _norm(x, w[p + "norm1"], eps)
            if layer["type"] == "latent_attention":
                y = _latent(h, w, p + "mix.", m, eps, kept)
            elif layer["type"] == "parallel":
                y = _grouped(h, w, p + "mix.left.", m["left"], torch.zeros(m["left"]["heads"], device="cuda", dtype=f64))
                z, S = _state_space(h, w, p + "mix.right.", m["right"], eps)
                y = 0.5 * (_norm(y, w[p + "mix.left.out"], eps) + _norm(z, w[p + "mix.right.out"], eps))
                states.setdefault(f"state{i}", []).append(S)
            else:
                y = _grouped(h, w, p + "mix.left.", m["left"], w[p + "mix.left.sink"])
                z, S = _delta_rule(h, w, p + "mix.right.", m["right"], eps)
                y = m["left_scale"] * y + m["right_scale"] * z
                states.setdefault(f"state{i}", []).append(S)
            x = x + _norm(y, w[p + "norm1b"], eps)
            h = _norm(x, w[p + "norm2"], eps)
            h = torch.nn.functional.silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)
            x = x + _norm(h @ w[p + "mlp.down"].T, w[p + "norm2b"], eps)
        logits.append(_norm(x[-1], w["final.norm"], eps) @ w["head"].T)
    return {"tokens": None, "logits": torch.stack(logits), **{k: torch.stack(s) for k, s in states.items()}}


def exact(case, seed):
    """The step in 64 bits: logits, and the cache or the recurrences' states it leaves behind."""
    return _exact_saluzen(case, seed) if case["model"] == "saluzen" else _exact_uniform(case, seed)
