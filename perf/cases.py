"""The work this framework is used for, as cases that can be timed and checked.

Four kinds, all through the calls a host program makes:

* ``linear``      -- one Linear layer: int8 (row quantisation, product, bias) or bf16, one row to thousands.
* ``attention``   -- one layer's causal attention: a prompt from position 0, or one new position over a paged cache.
* ``char``        -- the character-level float32 decoder, operator for operator, with its re-read of a full context.
* ``gpt``, ``fabezen``, ``topidra`` -- a decoder: reading prompts (``new`` = 0), or generating ``new`` tokens greedily.

Sizes are those of the benchmark and the tests, and odd ones around them.  Decoders are cut to a few layers: their layers are alike.
Weights are random, but the next-token distribution is peaked as a trained model's is (the head is correlated with the embedding
through a permutation), so that greedy tokens do not hang on the last bit of a logit.

``exact`` states the same arithmetic in float64 with plain torch operators.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from nn_b200 import native as N
from nn_b200.device import Device
from nn_b200.fabezen import Fabezen, FabezenConfig
from nn_b200.gpt import GptConfig, GptW8A8
from nn_b200.gpt_f32 import GptF32
from nn_b200.topidra import Topidra, TopidraConfig

VOCAB = 32000
u64, i64 = C.c_uint64, C.c_int64
_device = None


def device() -> Device:
    global _device
    if _device is None:
        _device = Device(0)
    return _device


# ------------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a prompt's rows through one int8 Linear: the benchmark's headline product, float activations in, float out
        {"name": "linear int8 8192 rows", "kind": "linear", "dtype": "int8", "rows": 8192, "k": 4096, "n": 4096, "in": "f32", "out": "f32"},
        # the few rows of a decoding step through one wide bf16 Linear: the weights are read once
        {"name": "linear bf16 8 rows", "kind": "linear", "dtype": "bf16", "rows": 8, "k": 4096, "n": 14336, "in": "bf16", "out": "bf16"},
        # the attention of one layer over prompts, and over a full paged cache for one new position
        {"name": "attention prompt 2048", "kind": "attention", "batch": 8, "heads": 32, "length": 2048, "step": False},
        {"name": "attention step 4096", "kind": "attention", "batch": 64, "heads": 32, "length": 4096, "step": True},
        # the character-level decoder of the samples: one sequence, tiny layers, every launch counts; the context fills once
        {"name": "char generate", "kind": "char", "batch": 1, "prompt": 32, "new": 128},
        # an interactive user of the int8 decoder: one sequence, a short prompt
        {"name": "gpt generate 1", "kind": "gpt", "batch": 1, "prompt": 32, "new": 64, "width": 2048, "heads": 16, "ff": 8192, "layers": 4},
        # serving a full batch
        {"name": "gpt generate 64", "kind": "gpt", "batch": 64, "prompt": 512, "new": 128, "width": 2048, "heads": 16, "ff": 8192, "layers": 4},
        # reading prompts of a length that fits no tile
        {"name": "gpt prompt 13x777", "kind": "gpt", "batch": 13, "prompt": 777, "new": 0, "width": 2048, "heads": 16, "ff": 8192, "layers": 4},
        # the decoder of delta rules and latent attention: prompts read in two portions, and a full batch decoding
        {"name": "fabezen prompt 16x1000", "kind": "fabezen", "batch": 16, "prompt": 1000, "new": 0, "width": 2048, "heads": 16, "ff": 5632, "window": 512,
         "layers": "dcl"},
        {"name": "fabezen generate 64", "kind": "fabezen", "batch": 64, "prompt": 128, "new": 64, "width": 2048, "heads": 16, "ff": 5632, "window": 512,
         "layers": "dcl"},
        # the decoder of linear and windowed attention: the same, the second with few sequences of an odd length
        {"name": "topidra prompt 16x1000", "kind": "topidra", "batch": 16, "prompt": 1000, "new": 0, "width": 2048, "heads": 16, "ff": 5632, "window": 512,
         "layers": "lagl"},
        {"name": "topidra generate 7", "kind": "topidra", "batch": 7, "prompt": 45, "new": 64, "width": 2048, "heads": 16, "ff": 5632, "window": 512,
         "layers": "lagl"},
    ]


def draw(rng):
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["linear", "linear", "attention", "attention", "char", "gpt", "gpt", "gpt", "fabezen", "fabezen", "topidra", "topidra"])
    if kind == "linear":
        dtype = rng.choice(["int8", "bf16"])
        return {"kind": kind, "dtype": dtype, "rows": spread(1, 8192), "k": 16 * spread(16, 320), "n": 8 * spread(64, 600),
                "in": "bf16" if dtype == "bf16" else rng.choice(["f32", "bf16"]), "out": rng.choice(["f32", "bf16"])}
    if kind == "attention":
        step = rng.random() < 0.5
        batch, heads = spread(1, 64 if step else 8), rng.choice([8, 16, 32])
        return {"kind": kind, "batch": batch, "heads": heads, "length": spread(64, 4096 if step else 2048), "step": step}
    if kind == "char":
        return {"kind": kind, "batch": rng.choice([1, 2, 3]), "prompt": spread(4, 120), "new": spread(32, 128)}
    width, heads = rng.choice([(1024, 8), (1024, 16), (2048, 16)])
    read = rng.random() < 0.5
    batch, prompt, new = (spread(1, 16), spread(33, 1000), 0) if read else (spread(1, 64), spread(8, 400), spread(16, 96))
    case = {"kind": kind, "batch": batch, "prompt": prompt, "new": new, "width": width, "heads": heads}
    if kind == "gpt":
        return {**case, "ff": 4 * width, "layers": rng.choice([2, 3, 4])}
    return {**case, "ff": 11 * width // 4, "window": rng.choice([128, 512]),
            "layers": rng.choice(["dcl", "ddl", "cl", "dc"] if kind == "fabezen" else ["lal", "lagl", "gl", "la"])}


# ------------------------------------------------------------------------------------------------------------------ inputs
class Rand:
    """Normal and uniform values on the GPU, one stream per seed."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed * 7919 + 17)

    def normal(self, *shape, std=1.0, mean=0.0):
        x = torch.randn(shape, generator=self.g, device="cuda")
        return x.mul_(std).add_(mean)

    def ids(self, *shape, bound):
        return torch.randint(0, bound, shape, generator=self.g, device="cuda").cpu().numpy().astype(np.int32)

    def permutation(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")


def _bits(t: torch.Tensor) -> np.ndarray:
    return t.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)


def _peaked_head(r: Rand, embed: torch.Tensor, std: float) -> torch.Tensor:
    """[vocab, width]: the row of a token's successor (a random permutation) leans towards the token's embedding."""
    V, D = embed.shape
    head = r.normal(V, D)
    after = r.permutation(V)
    head[after] += 28.0 / math.sqrt(D) * embed / embed.square().mean().sqrt()
    return head.mul_(std)


def _gpt_config(c) -> GptConfig:
    if c["kind"] == "char":
        return GptConfig(vocab=96, dim=128, heads=4, layers=4, ff_dim=512, context=128)
    return GptConfig(vocab=VOCAB, dim=c["width"], heads=c["heads"], layers=c["layers"], ff_dim=c["ff"], context=c["prompt"] + max(c["new"], 1))


def _gpt_weights(cfg: GptConfig, r: Rand) -> dict:
    """Float tensors on the GPU under the decoder's names."""
    D, FF, V = cfg.dim, cfg.ff_dim, cfg.vocab
    std = 0.02 if D > 128 else 0.08
    w = {"tok": r.normal(V, D), "pos": r.normal(cfg.context, D, std=0.02), "lnf_g": r.normal(D, std=0.05, mean=1.0), "lnf_b": r.normal(D, std=0.05),
         "head_b": r.normal(V, std=0.01)}
    w["head_w"] = _peaked_head(r, w["tok"], std).t().contiguous()
    for i in range(cfg.layers):
        p = f"l{i}."
        w.update({p + "ln1_g": r.normal(D, std=0.05, mean=1.0), p + "ln1_b": r.normal(D, std=0.05), p + "ln2_g": r.normal(D, std=0.05, mean=1.0),
                  p + "ln2_b": r.normal(D, std=0.05), p + "qkv_w": r.normal(D, 3 * D, std=std), p + "qkv_b": r.normal(3 * D, std=0.01),
                  p + "out_w": r.normal(D, D, std=std), p + "out_b": r.normal(D, std=0.01), p + "ff1_w": r.normal(D, FF, std=std),
                  p + "ff1_b": r.normal(FF, std=0.01), p + "ff2_w": r.normal(FF, D, std=std), p + "ff2_b": r.normal(D, std=0.01)})
    return w


def _block_config(c) -> dict:
    width, heads, ff = c["width"], c["heads"], c["ff"]
    dim = width // heads
    layers = []
    for kind in c["layers"]:
        if kind == "d":
            layer = {"type": "delta", "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": dim, "vdim": dim, "conv": 4}}
        elif kind == "c":
            layer = {"type": "channel_delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": dim, "vdim": dim, "conv": 4}}
        elif c["kind"] == "fabezen":
            layer = {"type": "latent_attention",
                     "mixer": {"heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "q_rank": 3 * width // 4, "kv_rank": 512, "scale": (1.5 * dim) ** -0.5,
                               "mask": {"size": c["window"]}, "rot": {"base": 10000.0, "dims": dim // 2}}}
        elif kind == "l":
            layer = {"type": "lightning", "mixer": {"heads": heads, "dim": dim, "vdim": dim, "decay": [1.0 - 2.0 ** (-2 - 8 * i / heads) for i in range(heads)]}}
        else:
            layer = {"type": "attention", "mixer": {"heads": heads, "kv_heads": heads if kind == "a" else heads // 4, "dim": dim, "vdim": dim,
                                                    "scale": dim ** -0.5, "mask": {"size": c["window"]}}}
        layers.append({**layer, "mlp": {"kind": "dense", "ff": ff}})
    cfg = {"architecture": c["kind"].capitalize(), "vocab": VOCAB, "width": width, "layers": layers, "norm": {"eps": 1e-5}}
    if c["kind"] == "fabezen":
        cfg.update(residual_mult=0.5, embedding={"scale": 1.0, "bigram": {"buckets": 32768, "mul_prev": 1009, "mul_cur": 31}})
    return cfg


def _block_weights(c, r: Rand) -> dict:
    """bf16 tensors on the GPU under the decoder's names."""
    cfg = _block_config(c)
    shapes = (FabezenConfig if c["kind"] == "fabezen" else TopidraConfig).from_dict(cfg).tensor_shapes()
    w = {}
    for name, shape in shapes.items():
        shape = tuple(c["width"] // c["heads"] if s is None else s for s in shape)
        last = name.rsplit(".", 1)[-1]
        if last in ("norm1b", "norm2b"):                     # gains after a sublayer are small in a deep model
            x = r.normal(*shape, std=0.03, mean=0.3)
        elif "norm" in last:
            x = r.normal(*shape, std=0.1, mean=1.0)
        elif last in ("A_log", "dt_bias"):
            x = r.normal(*shape, mean=-2.0)
        elif name == "head":
            x = _peaked_head(r, w["embed"].float(), c["width"] ** -0.5)
        elif name in ("embed", "bigram") or last == "sink":
            x = r.normal(*shape)
        else:
            x = r.normal(*shape, std=shape[-1] ** -0.5)
        w[name] = x.to(torch.bfloat16)
    return w


def _linear_inputs(c, r: Rand):
    w, b = r.normal(c["k"], c["n"], std=0.02), r.normal(c["n"], std=0.01)
    x = r.normal(c["rows"], c["k"])
    return w, b, x if c["in"] == "f32" else x.to(torch.bfloat16)


def _attention_inputs(c, r: Rand):
    """q, k, v [batch, length or 1, heads, 128]; the pages of a cache lie in any order."""
    B, H, L = c["batch"], c["heads"], c["length"]
    q = r.normal(B, 1 if c["step"] else L, H, 128).to(torch.bfloat16)
    k, v = (r.normal(B, L, H, 128).to(torch.bfloat16) for _ in range(2))
    return q, k, v


# ------------------------------------------------------------------------------------------------------------------ prepared state
class State:
    """What the program keeps between calls; `close` gives back what the library allocated."""

    def __init__(self, case, **kept):
        self.case = case
        self.__dict__.update(kept)

    def __del__(self):
        for name, handle in getattr(self, "handles", ()):
            try:
                N.call(name, handle)
            except Exception:
                pass
        if getattr(self, "model", None) is not None and hasattr(self.model, "close"):
            try:
                self.model.close()
            except Exception:
                pass


PAGE = 64


def prepare(case, seed):
    r, dev, c = Rand(seed), device(), case
    if c["kind"] == "linear":
        w, b, x = _linear_inputs(c, r)
        h = C.c_void_p()
        out = torch.empty(c["rows"], c["n"], dtype=torch.float32 if c["out"] == "f32" else torch.bfloat16, device="cuda")
        if c["dtype"] == "int8":
            wh, bh = w.cpu().numpy(), b.cpu().numpy()
            N.call("ns_linear_create", dev.handle, c["k"], c["n"], N.NS_I8, wh.ctypes.data_as(C.POINTER(C.c_float)), bh.ctypes.data_as(C.POINTER(C.c_float)),
                   N.SPLIT_NONE, 1, 0, 1, C.byref(h))
        else:
            wh = _bits(w.t().contiguous())
            N.call("ns_linear_create_bf16", dev.handle, c["n"], c["k"], wh.ctypes.data_as(C.c_void_p), C.byref(h))
        s = State(c, linear=h, x=x, out=out, handles=[("ns_linear_destroy", h)])
        if c["dtype"] == "int8":
            s.q, s.scale = torch.empty(c["rows"], c["k"], dtype=torch.int8, device="cuda"), torch.empty(c["rows"], device="cuda")
        torch.cuda.synchronize()
        return s
    if c["kind"] == "attention":
        q, k, v = _attention_inputs(c, r)
        B, H, L = c["batch"], c["heads"], c["length"]
        s = State(c, q=q, out=torch.empty_like(q), handles=[])
        if c["step"]:
            pages = (L + PAGE - 1) // PAGE
            s.pages, s.table = pages, r.permutation(B * pages).to(torch.int32)
            s.pos = torch.zeros(1, dtype=torch.int32, device="cuda")
            cache = C.c_void_p()
            N.call("ns_kv_cache_create", dev.handle, B * pages, PAGE, H, 128, C.byref(cache))
            s.cache, s.handles = cache, [("ns_kv_cache_destroy", cache)]
            torch.cuda.synchronize()
            N.call("ns_kv_append", dev.handle, cache, u64(k.data_ptr()), u64(v.data_ptr()), i64(H * 128), u64(s.table.data_ptr()), pages, u64(s.pos.data_ptr()), B, L)
            dev.synchronize()
            s.pos.fill_(L - 1)
        else:
            s.k, s.v = k, v
        torch.cuda.synchronize()
        return s
    if c["kind"] in ("char", "gpt"):
        cfg = _gpt_config(c)
        w = {k: t.cpu().numpy() for k, t in _gpt_weights(cfg, r).items()}
        prompt = r.ids(c["batch"], c["prompt"], bound=cfg.vocab)
        if c["kind"] == "char":
            return State(c, prompt=prompt, model=GptF32(dev, cfg, w, batch=c["batch"], max_steps=cfg.context))
        model = GptW8A8(dev, cfg, w, c["batch"], max_prefill=c["prompt"])
    else:
        w = {k: t.view(torch.int16).cpu().numpy().view(np.uint16) for k, t in _block_weights(c, r).items()}
        prompt = r.ids(c["batch"], c["prompt"], bound=VOCAB)
        cfg = _block_config(c)
        model = (Fabezen if c["kind"] == "fabezen" else Topidra)(dev, (FabezenConfig if c["kind"] == "fabezen" else TopidraConfig).from_dict(cfg), w, batch=c["batch"],
                                                                max_prefill=512)
    ids, logits = torch.empty(c["batch"], dtype=torch.int32, device="cuda"), torch.empty(c["batch"], VOCAB, device="cuda")
    torch.cuda.synchronize()
    return State(c, prompt=prompt, model=model, ids=ids, logits=logits)


# ------------------------------------------------------------------------------------------------------------------ one pass
def run(s):
    c, dev = s.case, device()
    h = dev.handle
    if c["kind"] == "linear":
        out = N.NS_F32 if c["out"] == "f32" else N.NS_BF16
        if c["dtype"] == "int8":
            N.call("ns_quantize_rows_i8", h, u64(s.x.data_ptr()), N.NS_F32 if c["in"] == "f32" else N.NS_BF16, i64(c["rows"]), c["k"], u64(s.q.data_ptr()),
                   u64(s.scale.data_ptr()))
            N.call("ns_linear_forward", h, s.linear, u64(s.q.data_ptr()), u64(s.scale.data_ptr()), c["rows"], N.EPI_BIAS, u64(0), N.NS_F32, out,
                   u64(s.out.data_ptr()))
        else:
            N.call("ns_linear_forward", h, s.linear, u64(s.x.data_ptr()), u64(0), c["rows"], N.EPI_NONE, u64(0), N.NS_F32, out, u64(s.out.data_ptr()))
        return s.out
    if c["kind"] == "attention":
        B, H, L, scale = c["batch"], c["heads"], c["length"], C.c_float(128 ** -0.5)
        if c["step"]:
            N.call("ns_attention_decode", h, s.cache, u64(s.q.data_ptr()), i64(H * 128), u64(s.out.data_ptr()), i64(H * 128), u64(s.table.data_ptr()), s.pages,
                   u64(s.pos.data_ptr()), B, 1, scale)
        else:
            strides = (i64 * 3)(L * H * 128, 128, H * 128)
            N.call("ns_attention_prefill", h, u64(s.q.data_ptr()), u64(s.k.data_ptr()), u64(s.v.data_ptr()), u64(s.out.data_ptr()), B, H, L, 128, strides, strides,
                   strides, strides, scale, 1)
        return s.out
    if c["kind"] == "char":
        tokens, _, logits = s.model.generate(s.prompt, c["new"])
        return {"tokens": tokens, "logits": np.stack(logits)}
    if c["new"]:
        tokens, _ = s.model.generate(s.prompt, c["new"])
    else:
        s.model.prefill(s.prompt)
        N.call("ns_d2d_async", h, u64(s.ids.data_ptr()), u64(s.model.ids.ptr), u64(4 * c["batch"]))
        tokens = s.ids
    N.call("ns_d2d_async", h, u64(s.logits.data_ptr()), u64(s.model.logits.ptr), u64(4 * c["batch"] * VOCAB))
    return {"tokens": tokens, "logits": s.logits}


# ------------------------------------------------------------------------------------------------------------------ what it cannot do without
def _layer_work(c, kind):
    """(weights, multiply-adds per token besides them, cached values read per token and position in reach, state values per sequence) of a layer."""
    D, H, ff = c["width"], c["heads"], c["ff"]
    dim = D // H
    if kind == "gpt":
        return 4 * D * D + 2 * D * ff, 0, 2 * D, 0
    mlp = 3 * D * ff
    if kind == "d":
        return 4 * D * D + 2 * D * H + mlp, 4 * D * dim, 0, D * dim
    if kind == "c":
        return 4 * D * D + D * H + 2 * D * dim + 2 * dim * D + mlp, 4 * D * dim, 0, D * dim
    if c["kind"] == "fabezen":
        rank, rot = 512, dim // 2
        return (3 * D // 4) * D + (D + H * rot) * (3 * D // 4) + (rank + rot) * D + 2 * D * rank + D * D + mlp, 0, rank + rot, 0
    if kind == "l":
        return 5 * D * D + mlp, 2 * D * dim, 0, D * dim
    kv = D if kind == "a" else D // 4
    return 2 * D * D + 2 * D * kv + D * H + mlp, 0, 2 * kv, 0


def work(case):
    c = case
    if c["kind"] == "linear":
        el, m, k, n = (1 if c["dtype"] == "int8" else 2), c["rows"], c["k"], c["n"]
        return {"bytes": el * k * n + (4 if c["in"] == "f32" else 2) * m * k + (4 if c["out"] == "f32" else 2) * m * n, "flops": 2.0 * m * k * n}
    if c["kind"] == "attention":
        B, D, L = c["batch"], 128 * c["heads"], c["length"]
        if c["step"]:
            return {"bytes": 2.0 * B * D * (2 * L + 2), "flops": 4.0 * B * D * L}
        return {"bytes": 8.0 * B * D * L, "flops": 2.0 * B * D * L * (L + 1)}
    B, P, new = c["batch"], c["prompt"], c["new"]
    if c["kind"] == "char":
        D, FF, V, layers, el = 128, 512, 96, 4, 4
        weights = layers * (4 * D * D + 2 * D * FF)
        return {"bytes": float(el * new * (weights + D * V + B * V)), "flops": 2.0 * B * ((P + new - 1) * weights + new * D * V)}
    layers = ["gpt"] * c["layers"] if c["kind"] == "gpt" else list(c["layers"])
    el, D = (1 if c["kind"] == "gpt" else 2), c["width"]
    passes = max(new, 1)                                     # the prompt's pass and one per token after the first
    bytes_, flops = float(passes * (el * D * VOCAB + 4 * B * VOCAB)), 2.0 * passes * B * D * VOCAB
    tokens = P + passes - 1
    for kind in layers:
        weights, extra, cached, state = _layer_work(c, kind)
        reach = [min(t, c.get("window", t)) for t in range(1, tokens + 1)]
        rows = float(sum(reach[P:]))                         # cached rows the decoding steps read
        heads = c["heads"] if kind == "l" and c["kind"] == "fabezen" else 1
        bytes_ += passes * el * weights + 2.0 * B * cached * (rows + tokens) + 8.0 * B * state * passes
        flops += 2.0 * B * (tokens * (weights + extra) + sum(reach) * cached * heads * (1 if heads == 1 else 2))
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times what `run` is away from `exact`: a rounding that falls the other way (int8 steps, bf16 steps), sums in another order."""
    c = case
    if c["kind"] == "linear" and c["dtype"] == "int8" and c["out"] == "f32":
        return {"rel": 1.5e-4, "max": 1e-2}
    if c["kind"] in ("linear", "attention"):
        return {"rel": 8e-3}
    if c["kind"] == "char":
        return {"rel": 3e-6, "max": 1e-4}
    return {"rel": 0.03 if c["kind"] == "gpt" else 0.012, "max": 0.4, "differ": 0.01}


# ------------------------------------------------------------------------------------------------------------------ the same in 64 bits
def _quantised(x):
    """Rows as int8 values times their scale."""
    s = x.abs().amax(-1, keepdim=True) / 127
    s = torch.where(s > 0, s, torch.ones_like(s))
    return (x / s).round().clamp(-127, 127) * s


def _norm(x, g, b, eps):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), g, b, eps)


def _rms(x, w, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt() * w


def _softmax_attention(q, k, v, scale, window=None, sink=None):
    """q [B, T, H, d], k, v [B, T, G, d] -> [B, T, H * dv], causal."""
    B, T, H, _ = q.shape
    rep = H // k.shape[2]
    k, v = (t.repeat_interleave(rep, 2).transpose(1, 2) for t in (k, v))
    i = torch.arange(T, device=q.device)
    back = i[:, None] - i[None, :]
    hidden = (back < 0) | (back >= (window or T))
    out = []
    for b in range(B):
        s = (q[b].transpose(0, 1) @ k[b].transpose(-1, -2)).mul_(scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, T, 1)], -1).softmax(-1)[..., :-1]
        else:
            s = s.softmax(-1)
        out.append((s @ v[b]).transpose(0, 1).reshape(T, -1))
    return torch.stack(out)


def _gpt64(w, cfg, tokens, quant):
    """Residual stream after the last norm [B, T, D]."""
    B, T = tokens.shape
    act = _quantised if quant else (lambda x: x)
    linear = lambda x, p: act(x) @ w[p + "_w"] + w[p + "_b"]
    x = w["tok"][tokens] + w["pos"][:T]
    for i in range(cfg.layers):
        p = f"l{i}."
        qkv = linear(_norm(x, w[p + "ln1_g"], w[p + "ln1_b"], cfg.eps), p + "qkv").reshape(B, T, 3, cfg.heads, -1)
        a = _softmax_attention(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], cfg.head_dim ** -0.5)
        x = x + linear(a, p + "out")
        f = linear(_norm(x, w[p + "ln2_g"], w[p + "ln2_b"], cfg.eps), p + "ff1")
        x = x + linear(torch.nn.functional.gelu(f, approximate="tanh"), p + "ff2")
    return _norm(x, w["lnf_g"], w["lnf_b"], cfg.eps)


def _short_conv(x, taps):
    n, T = taps.shape[1], x.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return torch.nn.functional.silu(sum(padded[:, j:j + T] * taps[:, j] for j in range(n)))


def _unit(x):
    return x * (x.square().sum(-1, keepdim=True) + 1e-6).rsqrt()


def _rotate(x, base, dims):
    """Neighbouring pairs of the last axis; x [B, T, ..., dims]."""
    T = x.shape[1]
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    a = (torch.arange(T, dtype=torch.float64, device=x.device)[:, None] * f).reshape((T,) + (1,) * (x.dim() - 3) + (dims // 2,))
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2)


def _mixer64(h, w, p, layer, eps):
    m, t = layer["mixer"], (lambda n: w[p + "mix." + n])
    B, T, _ = h.shape
    H, dim, vdim = m["heads"], m["dim"], m["vdim"]
    if layer["type"] == "attention":
        G = m["kv_heads"]
        q = _rms(h @ t("q").T, t("q.norm"), eps).reshape(B, T, H, dim)
        k = _rms(h @ t("k").T, t("k.norm"), eps).reshape(B, T, G, dim)
        o = _softmax_attention(q, k, (h @ t("v").T).reshape(B, T, G, vdim), m["scale"], m["mask"]["size"], t("sink"))
        return (o.reshape(B, T, H, vdim) * torch.sigmoid(h @ t("g").T)[..., None]).flatten(2) @ t("o").T
    if layer["type"] == "latent_attention":
        rank, rd, rot = m["kv_rank"], m["rot_dim"], m["rot"]
        q = (_rms(h @ t("dq").T, t("dq.norm"), eps) @ t("uq").T).reshape(B, T, H, dim + rd)
        down = h @ t("dkv").T
        cl = _rms(down[..., :rank], t("dkv.norm"), eps)
        k_rot = _rotate(down[..., rank:], rot["base"], rot["dims"])[:, :, None].expand(B, T, H, rd)
        q = torch.cat([q[..., :dim], _rotate(q[..., dim:], rot["base"], rot["dims"])], -1)
        k = torch.cat([(cl @ t("uk").T).reshape(B, T, H, dim), k_rot], -1)
        o = _softmax_attention(q, k, (cl @ t("uv").T).reshape(B, T, H, vdim), m["scale"], m["mask"]["size"])
        return o @ t("o").T
    s = torch.zeros(B, H, dim, vdim, dtype=torch.float64, device=h.device)
    o = torch.empty(B, T, H, vdim, dtype=torch.float64, device=h.device)
    if layer["type"] == "lightning":
        q, k, v = (torch.nn.functional.silu(h @ t(n).T).reshape(B, T, H, -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=torch.float64, device=h.device)[:, None, None]
        for i in range(T):
            s = s.mul_(decay).addcmul_(k[:, i, :, :, None], v[:, i, :, None, :])
            o[:, i] = (q[:, i, :, None, :] @ s).squeeze(2)
        return (_rms(o.flatten(2), t("norm"), eps) * torch.sigmoid(h @ t("g").T)) @ t("o").T
    rep = H // m["kv_heads"]
    q, k, v = (_short_conv(h @ t(n).T, t(n + ".conv")).reshape(B, T, -1, vdim if n == "v" else dim) for n in "qkv")
    q, k = (_unit(x).repeat_interleave(rep, 2) for x in (q, k))
    q = q * dim ** -0.5
    beta = torch.sigmoid(h @ t("b").T)
    if layer["type"] == "delta":
        a = (h @ t("a").T + t("dt_bias"))[..., None]
        gate = torch.nn.functional.silu(h @ t("g").T)
    else:
        a = ((h @ t("a1").T) @ t("a2").T + t("dt_bias")).reshape(B, T, H, dim)
        gate = torch.sigmoid((h @ t("g1").T) @ t("g2").T)
    decay = torch.exp(-torch.exp(t("A_log"))[:, None] * torch.nn.functional.softplus(a))
    for i in range(T):
        s = s.mul_(decay[:, i, :, :, None])
        seen = (k[:, i, :, None, :] @ s).squeeze(2)
        s = s.addcmul_(k[:, i, :, :, None], (beta[:, i, :, None] * (v[:, i] - seen))[:, :, None, :])
        o[:, i] = (q[:, i, :, None, :] @ s).squeeze(2)
    return (_rms(o, t("norm"), eps) * gate.reshape(B, T, H, vdim)).flatten(2) @ t("o").T


def _block64(w, cfg, tokens):
    eps, fab = cfg["norm"]["eps"], cfg["architecture"] == "Fabezen"
    x = w["embed"][tokens]
    if fab:
        b = cfg["embedding"]["bigram"]
        rows = torch.full_like(tokens, b["buckets"])
        rows[:, 1:] = (tokens[:, :-1] * b["mul_prev"] + tokens[:, 1:] * b["mul_cur"]) % b["buckets"]
        x = x * cfg["embedding"]["scale"] + w["bigram"][rows]
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        y = _mixer64(_rms(x, w[p + "norm1"], eps), w, p, layer, eps)
        x = x + (cfg["residual_mult"] * y if fab else _rms(y, w[p + "norm1b"], eps))
        h = _rms(x, w[p + "norm2"], eps)
        g = h @ w[p + "mlp.gate"].T
        g = torch.nn.functional.gelu(g, approximate="tanh") if fab else torch.relu(g)
        y = (g * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        x = x + (cfg["residual_mult"] * y if fab else _rms(y, w[p + "norm2b"], eps))
    return _rms(x, w["final.norm"], eps)


def _generate64(hidden, head, guess, prompt, n_new, context):
    """Greedy tokens [B, n_new] and their logits [n_new, B, V]: whole sequences at once, from guessed tokens until the guess holds
    (guess: the likely successor of every token [B])."""
    history, logits = prompt, []
    while len(logits) < n_new:
        keep = min(history.shape[1], context - 1) if not logits else context // 2
        count = min(n_new - len(logits), context - keep + 1)
        seq = torch.cat([history[:, -keep:], history.new_zeros(history.shape[0], count)], 1)
        for i in range(keep, keep + count):
            seq[:, i] = guess(seq[:, i - 1])
        for _ in range(count + 1):
            got = torch.cat([head(hidden(part[:, :-1])[:, keep - 1:]) for part in seq.split(8)])
            tokens = got.argmax(-1)
            if torch.equal(tokens, seq[:, keep:]):
                break
            seq[:, keep:] = tokens
        history = torch.cat([history, tokens], 1)
        logits += list(got.unbind(1))
    return history[:, -n_new:], logits


def exact(case, seed):
    r, c = Rand(seed), case
    if c["kind"] == "linear":
        w, b, x = (t.double() for t in _linear_inputs(c, r))
        if c["dtype"] == "int8":
            return _quantised(x) @ _quantised(w.t().contiguous()).t() + b
        return x @ w.to(torch.bfloat16).double()
    if c["kind"] == "attention":
        q, k, v = _attention_inputs(c, r)
        out = []
        for b in range(c["batch"]):
            qb, kb, vb = (t[b:b + 1].double() for t in (q, k, v))
            if c["step"]:
                p = (qb.transpose(1, 2) @ kb.permute(0, 2, 3, 1) * 128 ** -0.5).softmax(-1)
                out.append((p @ vb.transpose(1, 2)).transpose(1, 2))
            else:
                out.append(_softmax_attention(qb, kb, vb, 128 ** -0.5).reshape(qb.shape))
        return torch.cat(out)
    if c["kind"] in ("char", "gpt"):
        cfg = _gpt_config(c)
        quant = c["kind"] == "gpt"
        w = _gpt_weights(cfg, r)
        prompt = r.ids(c["batch"], c["prompt"], bound=cfg.vocab)
        if quant:
            w["tok"], w["pos"] = (w[n].to(torch.bfloat16) for n in ("tok", "pos"))
        w = {k: (_quantised(t.double().t().contiguous()).t() if quant and k.endswith("_w") else t.double()) for k, t in w.items()}
        hidden = lambda tokens: _gpt64(w, cfg, tokens, quant)
        head = lambda x: (_quantised(x) if quant else x) @ w["head_w"] + w["head_b"]
        embed, context = w["tok"], cfg.context
    else:
        cfg = _block_config(c)
        w = {k: t.double() for k, t in _block_weights(c, r).items()}
        prompt = r.ids(c["batch"], c["prompt"], bound=VOCAB)
        hidden = lambda tokens: _block64(w, cfg, tokens)
        matrix = w["embed" if c["kind"] == "fabezen" else "head"].t()
        head = lambda x: x @ matrix
        embed, context = w["embed"], 1 << 30
    tokens, logits = _generate64(hidden, head, lambda t: head(embed[t]).argmax(-1), torch.from_numpy(prompt).long().cuda(), max(c["new"], 1), context)
    if c["kind"] == "char":
        return {"tokens": None, "logits": torch.stack(logits)}
    return {"tokens": None, "logits": logits[-1]}
