"""Timed workloads of the engine: what a user's program runs through the public API (graph -> Planner -> Executor).

Every case is one plan with its weights and inputs resident in the executor's arena. One pass is what
`Runtime.run()` does: post one iteration and wait until its results are there. Five kinds of plan:

* decode  - one token for each sequence of a batch through a stack of decoder layers, against K/V caches;
* prefill - a prompt through a stack of decoder layers: causal attention from indices, with an additive mask tensor
            inside the fused attention stage, or as the reference example's matmul / softmax / matmul chain;
* ffn     - a feed-forward block Y = act(X W1) W2;
* rows    - what a language model does outside its matmuls: embedding lookup, position add, normalisations,
            activation, softmax, pooling;
* tiny    - the quickstart program: one elementwise operator on a small matrix.

Shapes are the benchmark configurations of this repository (7B- and 70B-shaped layers, the FFN blocks) and generic
ragged ones.
"""
import math

import numpy as np
import torch

import ark_b200 as ark
from ark_b200.ffn import build_ffn
from ark_b200.llama import LLAMA2_7B, LLAMA2_70B, LlamaConfig, decoder_layer, layer_weights

SHAPES = {"7b": LLAMA2_7B, "70b": LLAMA2_70B}
DTYPES = {"fp32": (ark.fp32, torch.float32), "fp16": (ark.fp16, torch.float16), "bf16": (ark.bf16, torch.bfloat16)}
STORED = {"FP32": torch.float32, "FP16": torch.float16, "BF16": torch.bfloat16, "INT32": torch.int32}
VOCAB = 32000


def listed():
    return [
        # one user's next token: latency of a single sequence (the decode benchmark's 7B shape)
        {"name": "decode_7b_1x2048", "kind": "decode", "shape": "7b", "dtype": "fp16", "batch": 1, "keys": 2048, "layers": 4},
        # a serving batch (the decode benchmark's 70B shape, grouped-query heads)
        {"name": "decode_70b_16x4096", "kind": "decode", "shape": "70b", "dtype": "bf16", "batch": 16, "keys": 4096, "layers": 2},
        # a half-full batch in the middle of a conversation
        {"name": "decode_7b_5x1337", "kind": "decode", "shape": "7b", "dtype": "bf16", "batch": 5, "keys": 1337, "layers": 2},
        # prompts (the prefill benchmark's two shapes)
        {"name": "prefill_7b_1x2048", "kind": "prefill", "shape": "7b", "dtype": "fp16", "batch": 1, "seq": 2048, "layers": 4,
         "attention": "causal"},
        {"name": "prefill_70b_4x1024", "kind": "prefill", "shape": "70b", "dtype": "bf16", "batch": 4, "seq": 1024, "layers": 2,
         "attention": "causal"},
        # the reference example's call: a mask tensor, attention as a chain of operators
        {"name": "prefill_7b_chain_1x1024", "kind": "prefill", "shape": "7b", "dtype": "fp16", "batch": 1, "seq": 1024, "layers": 1,
         "attention": "chain"},
        # a batch of prompts of different lengths: the padding is in the mask tensor
        {"name": "prefill_70b_padded_3x360", "kind": "prefill", "shape": "70b", "dtype": "bf16", "batch": 3, "seq": 360, "layers": 1,
         "attention": "mask"},
        # feed-forward blocks: the small one, the large one, and full precision (the default type of a tensor)
        {"name": "ffn_128_fp16", "kind": "ffn", "tokens": 128, "d_model": 1024, "d_ff": 4096, "dtype": "fp16", "act": "relu",
         "weights_nk": False},
        {"name": "ffn_4096_fp16", "kind": "ffn", "tokens": 4096, "d_model": 8192, "d_ff": 32768, "dtype": "fp16", "act": "gelu",
         "weights_nk": False},
        {"name": "ffn_300_fp32", "kind": "ffn", "tokens": 300, "d_model": 1024, "d_ff": 4096, "dtype": "fp32", "act": "relu",
         "weights_nk": True},
        # operators outside the matmuls, on the activations of a long batch
        {"name": "rows_8192x4096_bf16", "kind": "rows", "rows": 8192, "cols": 4096, "dtype": "bf16"},
        # the smallest call
        {"name": "tiny_64x64_fp16", "kind": "tiny", "rows": 64, "cols": 64, "dtype": "fp16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "prefill", "ffn", "ffn", "rows", "tiny"])
    if kind == "decode":
        return {"kind": kind, "shape": rng.choice(["7b", "70b"]), "dtype": rng.choice(["fp16", "bf16"]), "batch": _log_int(rng, 1, 16),
                "keys": _log_int(rng, 40, 4096), "layers": rng.choice([1, 2])}
    if kind == "prefill":
        attention = rng.choice(["causal", "causal", "mask", "chain"])
        shape = "7b" if attention == "chain" else rng.choice(["7b", "70b"])  # the chain has no grouped-query form
        batch = rng.choice([1, 1, 2, 3])
        seq = _log_int(rng, 33, (4096 if shape == "7b" else 2400) // batch // (4 if attention == "chain" else 1))
        seq = seq if attention == "causal" else (seq + 7) // 8 * 8  # rows of a mask tensor are whole 16-byte vectors
        return {"kind": kind, "shape": shape, "dtype": rng.choice(["fp16", "bf16"]), "batch": batch, "seq": seq, "layers": 1,
                "attention": attention}
    if kind == "ffn":
        dtype = rng.choice(["fp16", "fp16", "bf16", "bf16", "fp32"])
        # widths are multiples of 8 as weights usually are, one in five is not
        step = rng.choice([8, 8, 64, 128, 1])
        d_model = max(step, _log_int(rng, 256, 2048 if dtype == "fp32" or step == 1 else 8192) // step * step)
        tokens = _log_int(rng, 1, 512 if dtype == "fp32" or step == 1 else 4096)
        return {"kind": kind, "tokens": tokens, "d_model": d_model, "d_ff": rng.choice([2, 3, 4]) * d_model, "dtype": dtype,
                "act": rng.choice(["relu", "gelu", "silu"]), "weights_nk": rng.random() < 0.5}
    if kind == "rows":
        cols = _log_int(rng, 256, 8192) // 8 * 8  # the row operators take whole 16-byte vectors
        return {"kind": kind, "rows": _log_int(rng, 1, 8192), "cols": cols, "dtype": rng.choice(["fp32", "fp16", "bf16"])}
    return {"kind": kind, "rows": _log_int(rng, 1, 300), "cols": _log_int(rng, 8, 1024), "dtype": rng.choice(["fp32", "fp16", "bf16"])}


class _View:
    """Device memory of the executor's arena as a torch tensor; keeps the executor alive."""

    def __init__(self, ex, tensor):
        self.ex = ex
        kind = {"FP32": "<f4", "FP16": "<f2", "BF16": "<i2", "INT32": "<i4"}[tensor.dtype.name]
        self.__cuda_array_interface__ = {"shape": tuple(tensor.shape), "typestr": kind, "data": (ex.tensor_address(tensor), False),
                                         "version": 3}


def _view(ex, tensor):
    v = torch.as_tensor(_View(ex, tensor), device="cuda")
    return v.view(torch.bfloat16) if tensor.dtype is ark.bf16 else v


def _rope(seq, first, head_dim, theta=10000.0):
    """[1, seq, 1, head_dim], interleaved (cos, sin) pairs of positions first, first + 1, ..."""
    freq = theta ** (-torch.arange(0, head_dim, 2, device="cuda", dtype=torch.float64) / head_dim)
    angle = torch.outer(torch.arange(first, first + seq, device="cuda", dtype=torch.float64), freq)
    return torch.stack([angle.cos(), angle.sin()], -1).reshape(1, seq, 1, head_dim)


def _mask(batch, seq, padded, gen):
    """Additive causal mask; padded: one per sequence, which also hides the padding behind the sequence's own length."""
    m = torch.triu(torch.full((seq, seq), -math.inf, device="cuda"), 1).expand(batch if padded else 1, 1, seq, seq).clone()
    if padded:
        lengths = torch.randint(max(1, seq // 2), seq + 1, (batch,), generator=gen, device="cuda")
        m.masked_fill_((torch.arange(seq, device="cuda")[None, :] >= lengths[:, None])[:, None, None, :], -math.inf)
    return m


def _build(case, gen):
    """Adds the case's operators to the global model: ({tensor: values}, {name: output tensor}, the inputs' tensors by
    name: one dict for the call and one for each layer)."""
    ark.init()
    adt = DTYPES[case["dtype"]][0]

    def normal(shape, std=1.0, mean=0.0):
        return torch.randn(tuple(shape), generator=gen, device="cuda").mul_(std).add_(mean)

    if case["kind"] in ("decode", "prefill"):
        cfg = LlamaConfig(**SHAPES[case["shape"]])
        decode = case["kind"] == "decode"
        batch, seq, hd = case["batch"], 1 if decode else case["seq"], cfg.head_dim
        attention = "causal" if decode else case["attention"]
        x, rope = ark.tensor([batch * seq, cfg.dim], adt), ark.tensor([1, seq, 1, hd], adt)
        feeds = {x: normal(x.shape), rope: _rope(seq, case["keys"] if decode else 0, hd)}
        mask = None
        if attention != "causal":
            m = _mask(batch, seq, attention == "mask", gen)
            mask = ark.tensor(list(m.shape), adt)
            feeds[mask] = m
        h, named = x, [{"x": x, "rope": rope, "mask": mask}]
        for _ in range(case["layers"]):
            w = layer_weights(cfg, adt, 1)
            kc = vc = None
            if decode:
                kc, vc = (ark.tensor([batch, cfg.n_kv_heads, case["keys"], hd], adt) for _ in range(2))
                feeds[kc], feeds[vc] = normal(kc.shape), normal(vc.shape)
            h = decoder_layer(h, w, cfg, batch, seq, 0, 1, rope=rope, mask=mask, k_cache=kc, v_cache=vc,
                              causal=not decode and attention == "causal", fused_attention=attention == "mask")
            for k, t in w.items():
                if not (decode and k in ("wk", "wv")):  # a decode step finds its keys and values in the cache
                    feeds[t] = normal(t.shape, 0.05, 1.0) if "norm" in k else normal(t.shape, 0.02)
            named.append({**w, "kc": kc, "vc": vc})
        return feeds, {"hidden": h}, named
    if case["kind"] == "ffn":
        x, w1, w2, y = build_ffn(case["tokens"], case["d_model"], case["d_ff"], adt, act=case["act"], weights_nk=case["weights_nk"])
        return {x: normal(x.shape), w1: normal(w1.shape, 0.02), w2: normal(w2.shape, 0.02)}, {"y": y}, [{"x": x, "w1": w1, "w2": w2}]
    if case["kind"] == "rows":
        rows, cols = case["rows"], case["cols"]
        ids, table, pos = ark.tensor([rows], ark.int32), ark.tensor([VOCAB, cols], adt), ark.tensor([rows, cols], adt)
        gain, weight = ark.tensor([1, cols], adt), ark.tensor([cols], adt)
        x = ark.add(ark.reshape(ark.embedding(ids, table), [rows, cols]), pos)
        g = ark.gelu(ark.mul(ark.layernorm(x), gain))
        y, s = ark.rmsnorm(g, weight, residual=x)
        p = ark.cast(ark.softmax(y, scale=1.0 / math.sqrt(128)), ark.fp32) if adt is not ark.fp32 else ark.softmax(y, scale=1.0 / math.sqrt(128))
        pooled = ark.reduce_mean(s, axis=0)
        feeds = {ids: torch.randint(0, VOCAB, (rows,), generator=gen, device="cuda"), table: normal(table.shape), pos: normal(pos.shape, 0.1),
                 gain: normal(gain.shape, 0.05, 1.0), weight: normal(weight.shape, 0.05, 1.0)}
        named = {"ids": ids, "table": table, "pos": pos, "gain": gain, "weight": weight}
        return feeds, {"stream": s, "probabilities": p, "pooled": pooled}, [named]
    a, b = ark.tensor([case["rows"], case["cols"]], adt), ark.tensor([case["rows"], case["cols"]], adt)
    return {a: normal(a.shape), b: normal(b.shape)}, {"sum": ark.add(a, b)}, [{"a": a, "b": b}]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    feeds, outs, _ = _build(case, gen)
    ex = ark.Executor(torch.cuda.current_device(), 0, "case", str(ark.Planner(torch.cuda.current_device()).plan()), loop_mode=False)
    ex.compile()
    for t, values in feeds.items():
        v = values.to(STORED[t.dtype.name]).contiguous()
        torch.cuda.current_stream().synchronize()  # the executor copies on a stream of its own
        ex.tensor_write(t, v.data_ptr(), v.numel() * v.element_size(), is_d2d=True)
    ex.launch()
    return {"ex": ex, "outs": {k: _view(ex, t) for k, t in outs.items()}}


def run(state):
    state["ex"].run(1)
    state["ex"].wait()
    return state["outs"]


def _rotate(x, table):
    """x [batch, seq, heads, head_dim]; table [1, seq, 1, head_dim]."""
    a, b, cos, sin = x[..., 0::2], x[..., 1::2], table[..., 0::2], table[..., 1::2]
    return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).reshape(x.shape)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _rms(x, w, eps=1e-5):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer64(x, rope, mask, w, cfg, batch, seq, decode):
    hd, g = cfg.head_dim, cfg.n_heads // cfg.n_kv_heads
    h = _rms(x, w["attn_norm"], cfg.norm_eps)
    q = _rotate((h @ w["wq"].T).view(batch, seq, cfg.n_heads, hd), rope).transpose(1, 2)
    if decode:
        k, v = w["kc"], w["vc"]
    else:
        k = _rotate((h @ w["wk"].T).view(batch, seq, cfg.n_kv_heads, hd), rope).transpose(1, 2)
        v = (h @ w["wv"].T).view(batch, seq, cfg.n_kv_heads, hd).transpose(1, 2)
        if mask is None:
            mask = torch.triu(torch.full((seq, seq), -math.inf, device="cuda", dtype=torch.float64), 1)[None, None]
    o = torch.empty_like(q)
    for b in range(batch):
        for n in range(cfg.n_kv_heads):  # head by head: the scores of all heads at once would take gigabytes
            s = q[b, n * g:(n + 1) * g] @ k[b, n].T / math.sqrt(hd)
            if mask is not None:
                s = s + mask[min(b, mask.shape[0] - 1)]
            o[b, n * g:(n + 1) * g] = s.softmax(-1) @ v[b, n]
    x = x + o.transpose(1, 2).reshape(batch * seq, cfg.n_heads * hd) @ w["wo"].T
    h = _rms(x, w["ffn_norm"], cfg.norm_eps)
    return x + (torch.nn.functional.silu(h @ w["w1"].T) * (h @ w["w3"].T)) @ w["w2"].T


def exact(case, seed):
    """What run() returns for these inputs, in 64 bits throughout."""
    feeds, outs, named = _build(case, torch.Generator(device="cuda").manual_seed(int(seed)))
    feeds = {t: v.to(STORED[t.dtype.name]) for t, v in feeds.items()}  # the inputs as they are stored

    def wide(d):
        return {k: feeds[t].double() for k, t in d.items() if t in feeds}

    g = wide(named[0])
    if case["kind"] in ("decode", "prefill"):
        decode, x = case["kind"] == "decode", g["x"]
        for w in named[1:]:
            x = _layer64(x, g["rope"], g.get("mask"), wide(w), LlamaConfig(**SHAPES[case["shape"]]), case["batch"],
                         1 if decode else case["seq"], decode)
        return {"hidden": x}
    if case["kind"] == "ffn":
        w1, w2 = (g["w1"].T, g["w2"].T) if case["weights_nk"] else (g["w1"], g["w2"])
        act = {"relu": torch.relu, "gelu": _gelu, "silu": torch.nn.functional.silu}[case["act"]]
        return {"y": act(g["x"] @ w1) @ w2}
    if case["kind"] == "rows":
        x = g["table"][g["ids"].long()] + g["pos"]
        s = x + _gelu(torch.nn.functional.layer_norm(x, x.shape[-1:], eps=1e-5) * g["gain"])
        p = (_rms(s, g["weight"]) / math.sqrt(128)).softmax(-1)
        return {"stream": s, "probabilities": p, "pooled": s.mean(0, keepdim=True)}
    return {"sum": g["a"] + g["b"]}


def work(case):
    es = np.dtype(np.float32).itemsize if case["dtype"] == "fp32" else 2
    if case["kind"] in ("decode", "prefill"):
        cfg = LlamaConfig(**SHAPES[case["shape"]])
        decode = case["kind"] == "decode"
        batch, seq = case["batch"], 1 if decode else case["seq"]
        t, keys, n = batch * seq, case["keys"] if decode else case["seq"], case["layers"]
        hq, hkv, hd = cfg.n_heads, cfg.n_kv_heads, cfg.head_dim
        weights = cfg.dim * hd * (2 * hq + (0 if decode else 2 * hkv)) + 3 * cfg.dim * cfg.ffn_dim + 2 * cfg.dim
        pairs = keys if decode else (seq + 1) / 2  # keys per query row: a prompt's mask is causal
        nbytes = n * weights * es + 2 * t * cfg.dim * es + seq * hd * es
        if decode:
            nbytes += n * 2 * batch * hkv * keys * hd * es
        elif case["attention"] != "causal":
            nbytes += (batch if case["attention"] == "mask" else 1) * seq * seq * es
        return {"bytes": nbytes, "flops": n * (2.0 * t * weights + 4.0 * t * hq * pairs * hd)}
    if case["kind"] == "ffn":
        t, d, f = case["tokens"], case["d_model"], case["d_ff"]
        return {"bytes": (2 * t * d + 2 * d * f) * es, "flops": 4.0 * t * d * f}
    r, c = case["rows"], case["cols"]
    if case["kind"] == "rows":
        return {"bytes": r * 4 + 3 * c * es + r * c * (3 * es + 4), "flops": 40.0 * r * c}
    return {"bytes": 3 * r * c * es, "flops": float(r * c)}


def tolerance(case):
    # four times the distance from the same composition in float64, at the listed sizes: float32 block 1e-6; one block or
    # the row operators 3e-4 (fp16), 3e-3 (bf16); layer stacks, which round a dozen intermediates per layer, 1.5e-3
    # (fp16), 9e-3 (bf16), with single elements 8e-3 and 6e-2 off
    if case["kind"] == "tiny":
        return "exact"  # one rounding of one sum
    if case["dtype"] == "fp32":
        return {"rel": 5e-6, "max": 1e-4}
    stack = case["kind"] in ("decode", "prefill")
    if case["dtype"] == "fp16":
        return {"rel": 6e-3, "max": 0.035} if stack else {"rel": 1.5e-3, "max": 0.01}
    return {"rel": 0.03, "max": 0.25} if stack else {"rel": 1.2e-2, "max": 0.06}
