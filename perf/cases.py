"""Performance cases of the quantized-matmul path: the calls a serving program makes, over the range it makes them in.

A case is a dict of plain values.  Four kinds, each through the entry point that a model runs:

  linear   one ``GGUFLinearMethod.apply`` on an N x K matrix of one block type, `tokens` activation rows
  layer    the four linear layers of one decoder layer (q/k/v merged, attention output, gate/up merged, down), where
           the v and down matrices carry the larger block type, as the usual mixed files ("Q4_K_M") have it
  moe      one ``GGUFMoEMethod.apply``: routed experts, gate/up and down, routing weights, top-k sum
  embed    one embedding look-up in a quantized table

Weights are random blocks with the scale distributions of the benchmark configurations, activations are N(0, 1), router
logits N(0, 1).  The matrices of a state are what a loaded model holds; nothing else is kept from call to call.
"""
from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "vllm-gguf-plugin-prism_b200"))

from vllm_gguf_plugin.quantization import vocal_embeds  # noqa: E402
from vllm_gguf_plugin.quantization.fused_moe import GGUFMoEMethod  # noqa: E402
from vllm_gguf_plugin.quantization.linear import GGUFLinearMethod  # noqa: E402
from vllm_gguf_plugin.quantization.utils import SUPPORTED_QUANT_SIZES  # noqa: E402

NAMES = {"Q4_0": 2, "Q4_1": 3, "Q5_0": 6, "Q5_1": 7, "Q8_0": 8, "Q2_K": 10, "Q3_K": 11, "Q4_K": 12, "Q5_K": 13, "Q6_K": 14,
         "IQ2_XXS": 16, "IQ2_XS": 17, "IQ3_XXS": 18, "IQ1_S": 19, "IQ4_NL": 20, "IQ3_S": 21, "IQ2_S": 22, "IQ4_XS": 23, "IQ1_M": 29}
# byte offsets of the fp16 scales inside a block
SCALES = {"Q4_0": (0,), "Q4_1": (0, 2), "Q5_0": (0,), "Q5_1": (0, 2), "Q8_0": (0,), "Q2_K": (80, 82), "Q3_K": (108,), "Q4_K": (0, 2),
          "Q5_K": (0, 2), "Q6_K": (208,), "IQ2_XXS": (0,), "IQ2_XS": (0,), "IQ3_XXS": (0,), "IQ1_S": (0,), "IQ4_NL": (0,), "IQ3_S": (0,),
          "IQ2_S": (0,), "IQ4_XS": (0,), "IQ1_M": ()}
DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16}

MOST_WEIGHTS = 28672 * 8192            # values of one matrix
MOST_PRODUCTS = 1999 * 37888 * 3584    # multiply-adds of one pass


def listed():
    return [
        # the smallest call of a small model's decode step: latency and launches are all of it
        {"name": "decode small q8_0", "kind": "linear", "type": "Q8_0", "n": 3072, "k": 1024, "tokens": 1, "dtype": "float16"},
        # one token through a decoder layer of an 8B model in the most common mixed file
        {"name": "decode layer q4_k/q6_k", "kind": "layer", "type": "Q4_K", "type_v": "Q6_K", "hidden": 4096, "kv": 1024, "inter": 14336,
         "tokens": 1, "dtype": "float16"},
        # a few concurrent requests (or draft tokens), code-book weights
        {"name": "decode 4 iq4_xs", "kind": "linear", "type": "IQ4_XS", "n": 37888, "k": 3584, "tokens": 4, "dtype": "float16"},
        # batched decode of a lightly and of a well loaded server, an odd batch in the second
        {"name": "decode 8 q4_k", "kind": "linear", "type": "Q4_K", "n": 14336, "k": 4096, "tokens": 8, "dtype": "bfloat16"},
        {"name": "decode 45 q6_k", "kind": "linear", "type": "Q6_K", "n": 3584, "k": 18944, "tokens": 45, "dtype": "bfloat16"},
        # prefill chunks: an ordinary one, the largest one, and code-book weights of both sorts (2-bit MLP, 3-bit)
        {"name": "prefill 512 q4_k", "kind": "linear", "type": "Q4_K", "n": 14336, "k": 4096, "tokens": 512, "dtype": "float16"},
        {"name": "prefill 1999 q6_k", "kind": "linear", "type": "Q6_K", "n": 37888, "k": 3584, "tokens": 1999, "dtype": "bfloat16"},
        {"name": "prefill 128 iq2_xxs", "kind": "linear", "type": "IQ2_XXS", "n": 28672, "k": 8192, "tokens": 128, "dtype": "float16"},
        {"name": "prefill 300 iq3_s", "kind": "linear", "type": "IQ3_S", "n": 8192, "k": 28672, "tokens": 300, "dtype": "bfloat16"},
        # mixture of experts: a decode batch and a prefill chunk
        {"name": "moe decode 8 q4_0", "kind": "moe", "type": "Q4_0", "type_v": "Q4_0", "experts": 64, "top_k": 8, "hidden": 2048, "inter": 1024,
         "tokens": 8, "dtype": "float16"},
        {"name": "moe prefill 256 q4_0", "kind": "moe", "type": "Q4_0", "type_v": "Q4_0", "experts": 64, "top_k": 8, "hidden": 2048,
         "inter": 1024, "tokens": 256, "dtype": "float16"},
        # the token embedding of a prefill chunk
        {"name": "embed 1024 q6_k", "kind": "embed", "type": "Q6_K", "rows": 128256, "hidden": 4096, "tokens": 1024, "dtype": "bfloat16"},
    ]


def _log(rng, lo, hi, step=1):
    """Log-uniform between lo and hi, a multiple of `step`."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def _tokens(rng, hi):
    """One token in a third of the cases (plain decode), else anything up to `hi`."""
    return 1 if rng.random() < 0.33 else _log(rng, 2, max(2, hi))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["layer", "moe", "moe", "embed"])
    dtype = rng.choice(sorted(DTYPES))
    if kind == "linear":
        n = _log(rng, 512, 37888, rng.choice([1, 8, 64, 256]))
        k = min(_log(rng, 1024, 28672, 256), MOST_WEIGHTS // n // 256 * 256)
        return {"kind": kind, "type": rng.choice(sorted(NAMES)), "n": n, "k": k, "tokens": _tokens(rng, min(2048, MOST_PRODUCTS // (n * k))),
                "dtype": dtype}
    if kind == "layer":
        t, v = rng.choice([("Q4_K", "Q6_K"), ("Q4_K", "Q4_K"), ("Q5_K", "Q6_K"), ("Q3_K", "Q5_K"), ("Q2_K", "Q3_K"), ("Q8_0", "Q8_0"),
                           ("Q4_0", "Q4_0"), ("IQ4_XS", "Q5_K"), ("IQ3_S", "IQ4_XS")])
        hidden = _log(rng, 1024, 5120, 256)
        return {"kind": kind, "type": t, "type_v": v, "hidden": hidden, "kv": hidden // rng.choice([1, 2, 4, 8]),
                "inter": int(hidden * rng.uniform(2.5, 4)) // 256 * 256, "tokens": _tokens(rng, 512), "dtype": dtype}
    if kind == "moe":
        t, v = rng.choice([("Q4_0", "Q4_0"), ("Q4_K", "Q6_K"), ("Q8_0", "Q8_0"), ("Q5_K", "Q5_K"), ("Q2_K", "Q3_K"), ("Q6_K", "Q6_K")])
        experts = rng.choice([8, 16, 32, 64])
        hidden = _log(rng, 1024, 4096, 256)
        inter = min(_log(rng, 512, 4096, 256), max(256, MOST_WEIGHTS * 3 // (3 * experts * hidden) // 256 * 256))
        return {"kind": kind, "type": t, "type_v": v, "experts": experts, "top_k": rng.choice([2, 4, 8]), "hidden": hidden, "inter": inter,
                "tokens": _log(rng, 1, 1024), "dtype": dtype}
    return {"kind": kind, "type": rng.choice(sorted(NAMES)), "rows": _log(rng, 32000, 152064, 64), "hidden": _log(rng, 1024, 5120, 256),
            "tokens": _tokens(rng, 2048), "dtype": dtype}


# ---- inputs ------------------------------------------------------------------------------------------------


def _blocks(gen, name, rows, k):
    """uint8 [rows, bytes] of random blocks; the scales |N(0, 1)| * 0.01 (Q8_0: 0.002), everything else uniform bits."""
    per, size = SUPPORTED_QUANT_SIZES[NAMES[name]]
    nb = rows * (k // per)
    w = torch.randint(-(1 << 63), (1 << 63) - 1, ((nb * size + 7) // 8,), dtype=torch.int64, device="cuda", generator=gen)
    w = w.view(torch.uint8)[:nb * size].view(nb, size)

    def scale():
        return (torch.randn(nb, device="cuda", generator=gen).abs() * (0.002 if name == "Q8_0" else 0.01)).to(torch.float16)

    for at in SCALES[name]:
        w[:, at:at + 2] = scale().view(torch.uint8).view(nb, 2)
    if name == "Q8_0":
        w[:, 2:] = torch.randint(-127, 128, (nb, 32), dtype=torch.int8, device="cuda", generator=gen).view(torch.uint8)
    if name == "Q6_K":
        w[:, 192:208] = torch.randint(-32, 32, (nb, 16), dtype=torch.int8, device="cuda", generator=gen).view(torch.uint8)
    if name == "IQ1_M":   # the fp16 scale is spread over the top nibbles of four 16-bit words
        d = scale().view(torch.int16).to(torch.int32)
        sc = w[:, 48:56].contiguous().view(torch.int16).to(torch.int32)
        for i in range(4):
            sc[:, i] = (sc[:, i] & 0x0FFF) | (((d >> (4 * i)) & 0xF) << 12)
        w[:, 48:56] = sc.to(torch.int16).view(torch.uint8).view(nb, 8)
    return w.view(rows, (k // per) * size)


def _linear(gen, shards, k, dtype):
    """A loaded linear layer; `shards`: [(type, rows)], one for a plain layer, several for a merged one."""
    method, layer = GGUFLinearMethod(None), torch.nn.Module()
    rows = [r for _, r in shards]
    method.create_weights(layer, k, rows, k, sum(rows), dtype)
    ids = [None] if len(shards) == 1 else ["q", "k", "v"] if len(shards) == 3 else list(range(len(shards)))
    for sid, (name, r) in zip(ids, shards):
        layer.weight.weight_loader(layer.weight, _blocks(gen, name, r, k), sid)
        layer.weight_type.weight_loader(layer.weight_type, torch.tensor(NAMES[name]), sid)
    method.process_weights_after_loading(layer)
    return method, layer


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, tokens = DTYPES[case["dtype"]], case["tokens"]

    def acts(k):
        return torch.randn(tokens, k, device="cuda", generator=gen).to(dtype)

    if case["kind"] == "linear":
        method, layer = _linear(gen, [(case["type"], case["n"])], case["k"], dtype)
        return {"calls": [(method.apply, layer, acts(case["k"]))]}
    if case["kind"] == "layer":
        h, i, t, v = case["hidden"], case["inter"], case["type"], case["type_v"]
        calls = []
        for shards, k in (([(t, h), (t, case["kv"]), (v, case["kv"])], h), ([(t, h)], h), ([(t, i), (t, i)], h), ([(v, h)], i)):
            method, layer = _linear(gen, shards, k, dtype)
            calls.append((method.apply, layer, acts(k)))
        return {"calls": calls}
    if case["kind"] == "moe":
        e, h, i = case["experts"], case["hidden"], case["inter"]
        method, layer = GGUFMoEMethod(None), torch.nn.Module()
        method.create_weights(layer, e, h, i, dtype)
        for shard, name, rows, k in (("w1", case["type"], i, h), ("w3", case["type"], i, h), ("w2", case["type_v"], h, i)):
            param, kind = (layer.w2_weight, layer.w2_weight_type) if shard == "w2" else (layer.w13_weight, layer.w13_weight_type)
            param.weight_loader(param, _blocks(gen, name, e * rows, k).view(e, rows, -1), "experts", shard_id=shard, expert_id=0)
            kind.weight_loader(kind, torch.tensor(NAMES[name]), "experts", shard_id=shard)
        p = torch.randn(tokens, e, device="cuda", generator=gen).softmax(-1)
        weights, ids = p.topk(case["top_k"], dim=-1)
        return {"moe": method.apply, "layer": layer, "x": acts(h), "weights": weights, "ids": ids.to(torch.int32)}
    ids = torch.randint(0, case["rows"], (tokens,), device="cuda", generator=gen)
    return {"table": _blocks(gen, case["type"], case["rows"], case["hidden"]), "ids": ids, "type": NAMES[case["type"]],
            "hidden": case["hidden"], "dtype": dtype}


def run(state):
    if "calls" in state:
        return [apply(layer, x) for apply, layer, x in state["calls"]]
    if "moe" in state:
        return state["moe"](state["layer"], state["x"], state["weights"], state["ids"])
    return vocal_embeds._apply_gguf_embedding(state["ids"], state["table"], state["type"], state["hidden"], state["dtype"])


def work(case):
    def size(name, values):
        per, bytes_ = SUPPORTED_QUANT_SIZES[NAMES[name]]
        return values // per * bytes_

    t = case["tokens"]
    if case["kind"] == "linear":
        n, k = case["n"], case["k"]
        return {"bytes": size(case["type"], n * k) + 2 * t * (n + k), "flops": 2 * t * n * k}
    if case["kind"] == "layer":
        h, kv, i = case["hidden"], case["kv"], case["inter"]
        small, large = h * (h + kv) + h * h + 2 * h * i, h * kv + h * i
        rows = (h + 2 * kv) + h + 2 * i + h
        return {"bytes": size(case["type"], small) + size(case["type_v"], large) + 2 * t * (rows + 3 * h + i), "flops": 2 * t * (small + large)}
    if case["kind"] == "moe":
        e, k, h, i = case["experts"], case["top_k"], case["hidden"], case["inter"]
        used = e * (1 - (1 - k / e) ** t)     # experts that some token asks for
        one = size(case["type"], 2 * h * i) + size(case["type_v"], h * i)
        return {"bytes": int(used * one) + 4 * t * h + 8 * t * k, "flops": 6 * t * k * h * i}
    return {"bytes": size(case["type"], t * case["hidden"]) + 2 * t * case["hidden"] + 8 * t, "flops": t * case["hidden"]}


def tolerance(case):
    if case["kind"] == "embed":
        return "exact"
    if case["kind"] == "moe":
        # two products with an 8-bit re-quantization between them: a rounding of the first flips codes of the second
        return {"rel": 1e-2}
    return {"rel": 2e-3} if case["dtype"] == "float16" else {"rel": 4e-3}
