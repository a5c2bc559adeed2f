"""Performance cases of the quantized-inference path: what a user of this package has it do, through its public entry points.

Seven kinds of work, each over the sizes, types and options that are used in earnest:

* ``linear``    ``QuantizedLinear.forward`` of one projection shape (any row count, group size, act-order, bias);
* ``block``     the four fused projections of a transformer block, as a model that swapped in ``QuantizedLinear`` calls them;
* ``attend``    ``QuantizedKVCache.attend`` over the layers of a model: one token's attention over the packed cache;
* ``update``    ``QuantizedKVCache.update`` with a prompt, then token by token (the reference's contract: dense K / V come back);
* ``decode``    one ``DecodeStack`` step at a fixed context, replayed from a CUDA graph as ``bench.py`` and servers do;
* ``generate``  a prompt and a run of decode steps through ``DecodeStack``, launched from Python token by token;
* ``prompt``    ``DecodeStack.prefill`` of a long prompt, in one piece or in chunks.

``listed()`` are the cases to watch, ``draw(rng)`` gives more from the same ranges.  Weights, activations and caches are synthetic
(the distributions of ``bench.py``: INT4 codes with log-normal folded scales, N(0, 1) activations, keys with 1 % outlier channels).
"""

from __future__ import annotations

import math

import torch

from pare_b200 import KVCacheConfig, QuantConfig, QuantizedKVCache, QuantizedLinear
from pare_b200.decode import SHAPES, DecodeStack, synthetic_linear
from pare_b200.kv_cache import rope_table

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_DEVICE = "cuda"


def listed() -> list[dict]:
    return [
        # the smallest call: one projection, one token (the single-layer configuration of the benchmark)
        {"name": "linear_one_token", "kind": "linear", "n": 4096, "k": 4096, "layers": 1, "rows": 1, "dtype": "fp16",
         "group": 128, "act_order": False, "bias": False},
        # a large model's block, one token: weight streaming
        {"name": "block_70b_one_token", "kind": "block", "model": "llama-3-70b", "blocks": 1, "rows": 1, "dtype": "bf16",
         "act_order": False, "bias": False},
        # batched decode, sixteen sequences
        {"name": "block_8b_batch16", "kind": "block", "model": "llama-3.1-8b", "blocks": 1, "rows": 16, "dtype": "bf16",
         "act_order": False, "bias": False},
        # a GPTQ act-order model between decode and prompt sizes
        {"name": "block_8b_act_order_64", "kind": "block", "model": "llama-3.1-8b", "blocks": 1, "rows": 64, "dtype": "fp16",
         "act_order": True, "bias": False},
        # a ragged prompt through the linears of a model with odd sizes and biases
        {"name": "block_qwen_prompt_1531", "kind": "block", "model": "qwen2.5-7b", "blocks": 1, "rows": 1531, "dtype": "bf16",
         "act_order": False, "bias": True},
        # one sequence, all layers of a model: latency of the decode attention (rotary embedding inside)
        {"name": "attend_one_sequence_4k", "kind": "attend", "batch": 1, "ctx": 4096, "hq": 32, "hkv": 8, "bits": 4,
         "v_group": 0, "layers": 32, "dtype": "bf16", "rope": True},
        # a full batch of long contexts: cache streaming
        {"name": "attend_batch16_32k", "kind": "attend", "batch": 16, "ctx": 32768, "hq": 28, "hkv": 4, "bits": 4,
         "v_group": 0, "layers": 1, "dtype": "bf16", "rope": False},
        # 2-bit cache with values in 32-channel groups
        {"name": "attend_2bit_16k", "kind": "attend", "batch": 4, "ctx": 16384, "hq": 28, "hkv": 4, "bits": 2,
         "v_group": 32, "layers": 4, "dtype": "fp16", "rope": False},
        # the reference's cache contract: a prompt's tokens, then tokens one at a time, dense K / V every time
        {"name": "update_prompt_and_tokens", "kind": "update", "batch": 4, "hkv": 4, "ctx": 8191, "steps": 4, "bits": 4,
         "v_group": 0, "dtype": "fp16"},
        # the flagship of bench.py: one decode step of the 8B-shaped stack at 4096 cached tokens
        {"name": "decode_8b_one_sequence", "kind": "decode", "model": "llama-3.1-8b", "layers": 32, "batch": 1, "ctx": 4096,
         "dtype": "bf16"},
        # a short chat turn for four sequences, driven from Python (a few layers of the model)
        {"name": "generate_8b_batch4", "kind": "generate", "model": "llama-3.1-8b", "layers": 4, "batch": 4, "prompt": 200,
         "new": 40, "dtype": "bf16"},
        # a long ragged prompt
        {"name": "prompt_8b_4999", "kind": "prompt", "model": "llama-3.1-8b", "layers": 2, "batch": 1, "tokens": 4999,
         "chunks": 1, "dtype": "bf16"},
    ]


def _log(rng, lo: int, hi: int) -> int:
    """An integer between lo and hi, spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["linear", "linear", "linear", "block", "block", "attend", "attend", "attend", "update", "update",
                       "decode", "generate", "prompt", "prompt"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind == "linear":
        # most checkpoints: groups of 128 and sizes that are multiples of 64; some have smaller groups or ragged heights
        group = rng.choice([128, 128, 128, 128, 128, 128, 64, 32])
        k = _log(rng, 4, 112) * 128
        n = _log(rng, 8, 448) * 64
        if rng.random() < 0.2:
            n = _log(rng, 500, 8000)
        act_order = rng.random() < 0.2
        # layers outside the multiple-of-512 / groups-of-128 shapes are met at decode and short-prompt row counts
        rows = _log(rng, 1, 4096) if group == 128 and k % 512 == 0 else _log(rng, 1, 32)
        return {"kind": kind, "n": n, "k": k, "layers": rng.choice([1, 2, 3]), "rows": rows, "dtype": dtype, "group": group,
                "act_order": act_order, "bias": rng.random() < 0.3}
    if kind == "block":
        model = rng.choice(["llama-3.1-8b", "llama-3.1-8b", "qwen2.5-7b", "llama-3-70b"])
        return {"kind": kind, "model": model, "blocks": 1, "rows": _log(rng, 1, 1024 if model == "llama-3-70b" else 3000), "dtype": dtype,
                "act_order": rng.random() < 0.25, "bias": model == "qwen2.5-7b"}
    if kind == "attend":
        hkv = rng.choice([4, 8])
        hq = hkv * rng.choice([4, 7, 8])
        batch = _log(rng, 1, 16)
        ctx = _log(rng, 150, 32768)
        layers = max(1, min(32, (64 << 20) // (batch * hkv * ctx * 168)))
        return {"kind": kind, "batch": batch, "ctx": ctx, "hq": hq, "hkv": hkv, "bits": rng.choice([4, 4, 2]),
                "v_group": rng.choice([0, 0, 32]), "layers": layers, "dtype": dtype, "rope": rng.random() < 0.5}
    if kind == "update":
        batch, hkv = _log(rng, 1, 8), rng.choice([4, 8])
        ctx = _log(rng, 100, max(200, 150000 // (batch * hkv)))
        return {"kind": kind, "batch": batch, "hkv": hkv, "ctx": ctx, "steps": _log(rng, 1, 8), "bits": rng.choice([4, 4, 2, 8]),
                "v_group": rng.choice([0, 0, 32]), "dtype": dtype}
    if kind == "decode":
        model = rng.choice(["llama-3.1-8b", "qwen2.5-7b", "llama-3-70b"])
        return {"kind": kind, "model": model, "layers": 4 if model == "llama-3-70b" else rng.randrange(4, 17),
                "batch": rng.choice([1, 1, 2, 3, 4, 6, 8, 12, 16]), "ctx": _log(rng, 200, 16384), "dtype": dtype}
    if kind == "generate":
        return {"kind": kind, "model": rng.choice(["llama-3.1-8b", "qwen2.5-7b"]), "layers": rng.randrange(2, 7),
                "batch": rng.choice([1, 1, 2, 3, 4, 6, 8]), "prompt": _log(rng, 16, 1000), "new": _log(rng, 8, 64), "dtype": dtype}
    model = rng.choice(["llama-3.1-8b", "qwen2.5-7b"])
    batch = rng.choice([1, 1, 1, 2, 4])
    return {"kind": kind, "model": model, "layers": 1, "batch": batch, "tokens": _log(rng, 100, 8000 // batch),
            "chunks": rng.choice([1, 1, 1, 2, 3]), "dtype": dtype}


# ---- inputs -------------------------------------------------------------------------------------------------------------

def _layer(n: int, k: int, seed: int, group: int, act_order: bool, bias: bool, dtype) -> QuantizedLinear:
    """A random INT4 layer as the loaders of this package give it, on the GPU and switched to the kernels."""
    layer = synthetic_linear(n, k, seed=seed, device=_DEVICE, group_size=group)
    if act_order or bias:
        g = torch.Generator(device=_DEVICE).manual_seed(seed + 1)
        g_idx = None
        if act_order:   # a random permutation of the input channels, mapped to groups
            g_idx = torch.empty(k, dtype=torch.int32, device=_DEVICE)
            g_idx[torch.randperm(k, device=_DEVICE, generator=g)] = (torch.arange(k, device=_DEVICE) // group).to(torch.int32)
        b = 0.1 * torch.randn(n, device=_DEVICE, generator=g).to(dtype) if bias else None
        cfg = QuantConfig(bits=4, scheme="gptq" if act_order else "awq", group_size=group, act_order=act_order)
        layer = QuantizedLinear.from_tensors(layer.packed_weight, None, layer.scale, layer.zero, cfg, b, k, n, g_idx=g_idx)
        layer.use_kernel = True
    return layer


def _rows(shape, seed: int, dtype) -> torch.Tensor:
    g = torch.Generator(device=_DEVICE).manual_seed(seed)
    return torch.randn(*shape, device=_DEVICE, generator=g).to(dtype)


def _keys_values(batch: int, heads: int, tokens: int, seed: int, dtype):
    """N(0, 1) keys and values of head dimension 128, 1 % of the key channels ten times larger."""
    g = torch.Generator(device=_DEVICE).manual_seed(seed)
    k = torch.randn(batch, heads, tokens, 128, device=_DEVICE, generator=g, dtype=torch.float32).to(dtype)
    v = torch.randn(batch, heads, tokens, 128, device=_DEVICE, generator=g, dtype=torch.float32).to(dtype)
    k[..., torch.randperm(128, device=_DEVICE, generator=g)[:1]] *= 10.0
    return k, v


def _quiet_context(ctx: int, residual: int = 128, group: int = 32) -> int:
    """The context at or a little below ``ctx`` from which a few single-token steps compress nothing (a graph replays one step)."""
    over = max(0, ctx - residual) % group
    return ctx - max(0, over - (group - 4)) if ctx > residual else min(ctx, residual - 4)


def _capture(fn):
    """``fn`` warmed up and captured on one stream of its own; returns (graph, outputs)."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        fn()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = fn()
    return graph, out


def _projections(model: str):
    hidden, ffn, hq, hkv, d, _ = SHAPES[model]
    return [((hq + 2 * hkv) * d, hidden), (hidden, hq * d), (2 * ffn, hidden), (hidden, ffn)]   # q|k|v, o, gate|up, down


@torch.no_grad()
def prepare(case: dict, seed: int) -> dict:
    kind, dtype = case["kind"], _DTYPES[case["dtype"]]
    if kind in ("linear", "block"):
        if kind == "linear":
            shapes, group, biases = [(case["n"], case["k"])] * case["layers"], case["group"], [case["bias"]] * case["layers"]
        else:
            shapes, group = _projections(case["model"]) * case["blocks"], 128
            biases = [case["bias"], False, False, False] * case["blocks"]   # such models have them on q|k|v only
        layers = [_layer(n, k, seed * 1000 + 10 * i, group, case["act_order"], b, dtype) for i, ((n, k), b) in enumerate(zip(shapes, biases))]
        xs = [_rows((case["rows"], k), seed * 1000 + 10 * i + 5, dtype) for i, (_, k) in enumerate(shapes)]
        return {"kind": kind, "layers": layers, "xs": xs}
    if kind == "attend":
        n = case["layers"]
        ctx = _quiet_context(case["ctx"])
        cache = QuantizedKVCache(n, KVCacheConfig(bits=case["bits"], v_group_size=case["v_group"] or None), max_seq_len=ctx + 64)
        for i in range(n):
            cache.update(i, *_keys_values(case["batch"], case["hkv"], ctx, seed * 100 + i, dtype))
        q = _rows((n, case["batch"], case["hq"], 1, 128), seed * 100 + 90, dtype)
        k1 = _rows((n, case["batch"], case["hkv"], 1, 128), seed * 100 + 91, dtype)
        v1 = _rows((n, case["batch"], case["hkv"], 1, 128), seed * 100 + 92, dtype)
        row = rope_table(ctx + 1, 128, device=_DEVICE)[ctx].clone() if case["rope"] else None

        def step():
            return [cache.attend(i, q[i], k1[i], v1[i], rope=row) for i in range(n)]

        graph, out = _capture(step)
        # what comes back: the outputs, and the first layer's window with the token that was appended
        return {"kind": kind, "graph": graph, "out": [*out, cache._residual_k[0], cache._residual_v[0]], "keep": (cache, q, k1, v1, row)}
    if kind == "update":
        cfg = KVCacheConfig(bits=case["bits"], v_group_size=case["v_group"] or None)
        cache = QuantizedKVCache(1, cfg, max_seq_len=case["ctx"] + case["steps"])
        k, v = _keys_values(case["batch"], case["hkv"], case["ctx"] + case["steps"], seed, dtype)
        pieces = [(k[:, :, :case["ctx"]].contiguous(), v[:, :, :case["ctx"]].contiguous())]
        pieces += [(k[:, :, t:t + 1].contiguous(), v[:, :, t:t + 1].contiguous()) for t in range(case["ctx"], case["ctx"] + case["steps"])]
        return {"kind": kind, "cache": cache, "pieces": pieces}

    hidden = SHAPES[case["model"]][0]
    if kind == "decode":
        ctx = _quiet_context(case["ctx"])
        stack = DecodeStack(case["model"], dtype=dtype, n_layers=case["layers"], max_seq_len=ctx + 64, seed=seed * 100)
        stack.prefill_cache(case["batch"], ctx, seed=seed)
        x = _rows((case["batch"], hidden), seed * 100 + 90, dtype)
        graph, out = _capture(lambda: stack(x))
        return {"kind": kind, "graph": graph, "out": [out, stack.cache._residual_k[0], stack.cache._residual_v[0]], "keep": (stack, x)}
    if kind == "generate":
        stack = DecodeStack(case["model"], dtype=dtype, n_layers=case["layers"], max_seq_len=case["prompt"] + case["new"] + 64, seed=seed * 100)
        return {"kind": kind, "stack": stack, "x": _rows((case["batch"], case["prompt"], hidden), seed * 100 + 90, dtype),
                "tokens": list(_rows((case["new"], case["batch"], hidden), seed * 100 + 91, dtype))}
    stack = DecodeStack(case["model"], dtype=dtype, n_layers=case["layers"], max_seq_len=case["tokens"] + 64, seed=seed * 100)
    x = _rows((case["batch"], case["tokens"], hidden), seed * 100 + 90, dtype)
    return {"kind": kind, "stack": stack, "chunks": [c.contiguous() for c in x.chunk(case["chunks"], dim=1)]}


# ---- one pass -----------------------------------------------------------------------------------------------------------

@torch.no_grad()
def run(state: dict):
    kind = state["kind"]
    if kind in ("linear", "block"):
        return [layer(x) for layer, x in zip(state["layers"], state["xs"])]
    if kind in ("attend", "decode"):
        state["graph"].replay()
        return state["out"]
    if kind == "update":
        cache = state["cache"]
        cache.reset()
        for k, v in state["pieces"]:
            full = cache.update(0, k, v)
        return full
    stack = state["stack"]
    stack.cache.reset()
    if kind == "prompt":
        hidden = [stack.prefill(c) for c in state["chunks"]]
        return [*hidden, stack.cache._residual_k[0], stack.cache._residual_v[0]]
    out = [stack.prefill(state["x"])]
    steps = [stack(x) for x in state["tokens"]]   # one token of every sequence at a time (the token's embedding is the caller's)
    return [*out, torch.stack(steps), stack.cache._residual_k[0], stack.cache._residual_v[0]]


# ---- what a pass cannot do without --------------------------------------------------------------------------------------

def _linear_work(m: int, n: int, k: int, group: int = 128):
    """Nibbles, 16-bit scale and zero per group, activations in and out; two operations per product."""
    return n * k // 2 + 2 * n * (k // group) * 2 + m * k * 2 + m * n * 2, 2 * m * n * k


def _token_bytes(bits: int, v_group: int) -> int:
    """Bytes of one compressed token and KV head (D = 128, key groups of 32 tokens, fp32 scale and zero)."""
    return 2 * 128 * bits // 8 + 2 * 128 * 4 // 32 + 2 * 4 * (4 if v_group else 1)


def _compressed(total: int) -> int:
    return max(0, total - 128) // 32 * 32


def _attend_work(batch: int, ctx: int, hq: int, hkv: int, bits: int, v_group: int):
    n_c = _compressed(ctx)
    nbytes = batch * hkv * (n_c * _token_bytes(bits, v_group) + (ctx - n_c) * 512) + batch * hq * 128 * 4
    return nbytes, 4 * batch * hq * ctx * 128


def _block_work(model: str, rows: int):
    parts = [_linear_work(rows, n, k) for n, k in _projections(model)]
    return sum(p[0] for p in parts), sum(p[1] for p in parts)


def _prompt_work(model: str, batch: int, tokens: int):
    """One block over a prompt: its linears, causal attention (half of a square), keys and values into the cache."""
    _, _, hq, hkv, d, _ = SHAPES[model]
    nbytes, flops = _block_work(model, batch * tokens)
    nbytes += batch * hkv * (_compressed(tokens) * _token_bytes(4, 0) + min(tokens, 128) * 512)
    return nbytes, flops + 2 * batch * hq * tokens * tokens * d


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "linear":
        b, f = _linear_work(case["rows"], case["n"], case["k"], case["group"])
        return {"bytes": case["layers"] * b, "flops": case["layers"] * f}
    if kind == "block":
        b, f = _block_work(case["model"], case["rows"])
        return {"bytes": case["blocks"] * b, "flops": case["blocks"] * f}
    if kind == "attend":
        b, f = _attend_work(case["batch"], _quiet_context(case["ctx"]) + 2, case["hq"], case["hkv"], case["bits"], case["v_group"])
        return {"bytes": case["layers"] * b, "flops": case["layers"] * f}
    if kind == "update":
        # the prompt: read once, compressed, dense result written; every token: packed cache and window read, dense result written
        heads, per = case["batch"] * case["hkv"], _token_bytes(case["bits"], case["v_group"])
        total = 0
        for t in range(case["ctx"], case["ctx"] + case["steps"] + 1):
            n_c = _compressed(t)
            total += heads * (n_c * per + (t - n_c) * 512 + t * 512)
        return {"bytes": total + heads * case["ctx"] * 512, "flops": 0}
    hidden, _, hq, hkv, d, _ = SHAPES[case["model"]]
    if kind == "decode":
        b, f = _block_work(case["model"], case["batch"])
        ab, af = _attend_work(case["batch"], _quiet_context(case["ctx"]) + 2, hq, hkv, 4, 0)
        return {"bytes": case["layers"] * (b + ab), "flops": case["layers"] * (f + af)}
    if kind == "prompt":
        b, f = _prompt_work(case["model"], case["batch"], case["tokens"])
        return {"bytes": case["layers"] * b, "flops": case["layers"] * f}
    b, f = _prompt_work(case["model"], case["batch"], case["prompt"])
    sb, sf = _block_work(case["model"], case["batch"])
    for t in range(case["prompt"] + 1, case["prompt"] + case["new"] + 1):
        ab, af = _attend_work(case["batch"], t, hq, hkv, 4, 0)
        b, f = b + sb + ab, f + sf + af
    return {"bytes": case["layers"] * b, "flops": case["layers"] * f}


def tolerance(case: dict):
    """About four times what a 64-bit restatement of the path differs by (outputs of 16-bit types: their own rounding is most of it)."""
    kind, bf16 = case["kind"], case["dtype"] == "bf16"
    if kind == "update":
        return "exact"      # codes, scales, zeros and their reconstruction are defined to the bit
    if kind in ("linear", "block"):     # seen: 2.3e-3 / 2.9e-4
        return {"rel": 8e-3 if bf16 else 1.2e-3}
    if kind == "attend":                # seen: 1.7e-3 / 2.1e-4
        return {"rel": 7e-3 if bf16 else 1e-3}
    if kind == "prompt":                # seen: 1.2e-3 with single values off by 0.076 / 1.1e-4, 1.9e-3
        return {"rel": 5e-3, "max": 0.3} if bf16 else {"rel": 1e-3, "max": 0.04}
    # a chain of blocks with a rounding at every hand-over; rows whose residual stream nearly cancels magnify it (seen: 2.4e-3 /
    # 1.1e-3 with single values off by 0.02 / 0.03)
    return {"rel": 1.2e-2, "max": 0.5} if bf16 else {"rel": 4e-3, "max": 0.2}
