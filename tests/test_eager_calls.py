"""GPU: the functions that eager calls go through (csrc/eager.cpp)."""
import threading
import time

import numpy as np
import pytest
import torch

from gguf_b200 import capi, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"


def weight(t, n, k, seed=0):
    return torch.from_numpy(synth.make_weight(t, n, k, seed=seed)).to(DEV)


def merged_layer(types, rows, K, dtype=torch.float16):
    """A loaded q/k/v layer whose shards have the given block types, and its parts."""
    from vllm_gguf_plugin.quantization.linear import GGUFLinearMethod

    method, layer = GGUFLinearMethod(None), torch.nn.Module()
    method.create_weights(layer, K, rows, K, sum(rows), dtype)
    parts = [weight(t, r, K, seed=r) for t, r in zip(types, rows)]
    for sid, t, w in zip("qkv", types, parts):
        layer.weight.weight_loader(layer.weight, w, sid)
        layer.weight_type.weight_loader(layer.weight_type, torch.tensor(t), sid)
    method.process_weights_after_loading(layer)
    return method, layer, parts


def eager_call(kind):
    from vllm_gguf_plugin import native

    w, x = weight(12, 64, 256), torch.randn(1, 256, device=DEV).half()
    if kind == "linear":
        return lambda: native.linear(x, w, 12)
    if kind == "mul_mat":
        return lambda: native.mul_mat(w, x, 12, 64, capi.OP_GEMV)
    if kind == "embed":
        ids = torch.arange(4, device=DEV)
        return lambda: native.embed(ids, w, 12, 256, torch.float16)
    if kind == "linear_runs":
        _, layer, _ = merged_layer((12, 12, 14), [64, 32, 32], 2048)
        x2 = torch.randn(1, 2048, device=DEV).half()
        return lambda: native.linear_runs(x2, layer.weight, layer.weight.gguf_runs)
    w13, w2 = (torch.from_numpy(np.stack([synth.make_weight(2, 128, k, seed=e) for e in range(4)])).to(DEV) for k in (128, 64))
    ids, tw = torch.zeros(1, 2, dtype=torch.int32, device=DEV), torch.ones(1, 2, device=DEV)
    x3 = torch.randn(1, 128, device=DEV).half()
    return lambda: native.moe(x3, w13, w2, tw, ids, 2, 2, 1)


@pytest.mark.parametrize("kind", ["linear", "mul_mat", "embed", "linear_runs", "moe"])
def test_other_threads_run_while_a_call_waits_for_the_launch_queue(native_libs, kind):
    """Behind a kernel of about 0.6 s the queue fills up and a call waits for it to drain; other Python threads go on."""
    call = eager_call(kind)
    assert call() is not None
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    thread = threading.Thread(target=tick)
    thread.start()
    torch.cuda._sleep(1_200_000_000)
    t0 = time.perf_counter()
    for _ in range(4000):
        call()
    t1 = time.perf_counter()
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    assert capi.last_status() == 0
    seen = [t0, *(t for t in ticks if t0 <= t <= t1), t1]
    assert t1 - t0 > 0.2, "the queue never filled up"
    assert max(b - a for a, b in zip(seen, seen[1:])) < 0.5 * (t1 - t0)


# (operation, tokens, K): the one-launch and the two-launch GEMV, two vectors, the small-batch kernel, the tiled one, the GEMM
# on plain activations with whole tiles and with shared ones, the GEMV per routed expert
IN_FLIGHT = [("vec", "Q4_K", 1, 1024), ("vec", "Q6_K", 1, 8192), ("vec", "Q8_0", 2, 1024), ("vec", "Q4_K", 2, 8192), ("vec", "IQ4_XS", 5, 1024), ("mmq", "Q4_K", 8, 1024),
             ("mmq", "Q6_K", 40, 2048), ("dqmm", "IQ2_XXS", 300, 1024), ("dqmm", "IQ4_XS", 20, 4096), ("moe_vec", "Q4_0", 3, 1024)]


@pytest.mark.parametrize("eager", [True, False])
@pytest.mark.parametrize("case", IN_FLIGHT)
def test_products_of_weights_that_a_kernel_has_just_written(native_libs, case, eager):
    """Weights that come straight out of a kernel are read behind it, through the functions and through the operators."""
    from helpers import TYPES
    from vllm_gguf_plugin import ops

    kind, name, M, K = case
    t, N, E = TYPES[name], 4096, 4 if kind == "moe_vec" else 1
    ws = [weight(t, N * E, K, seed=s) for s in (1, 2)]
    x = torch.randn(M, K, device=DEV).half()
    ids = torch.arange(M * 2, device=DEV, dtype=torch.int32).view(M, 2) % E
    op = torch.ops._C_gguf

    def product(w):
        if kind == "moe_vec":
            return ops.ggml_moe_a8_vec(x, w.view(E, N, -1), ids, 2, t, N, M)
        if eager:
            return {"vec": ops.ggml_mul_mat_vec_a8, "mmq": ops.ggml_mul_mat_a8, "dqmm": ops.ggml_dequant_matmul}[kind](w, x, t, N)
        return {"vec": op.ggml_mul_mat_vec_a8, "mmq": op.ggml_mul_mat_a8, "dqmm": op.dequant_matmul}[kind](w, x, t, N)

    want = []
    for w in ws:
        torch.cuda.synchronize()
        want.append(product(w))
    buf = torch.empty_like(ws[0])
    torch.cuda.synchronize()
    got = []
    for i in range(40):
        buf.copy_(ws[i & 1])
        got.append(product(buf))
    torch.cuda.synchronize()
    assert capi.last_status() == 0
    assert all(torch.equal(y, want[i & 1]) for i, y in enumerate(got))


def test_first_product_behind_loading_reads_the_loaded_weights(native_libs):
    """A layer's products may read its weights ahead of the stream, so loading puts a kernel of its own behind the writes."""
    from vllm_gguf_plugin.quantization.linear import GGUFLinearMethod

    files = [weight(12, 8192, 1024, seed=s) for s in (1, 2)]
    x = torch.randn(1, 1024, device=DEV).half()
    want = [capi.mul_mat_vec_a8(w, x, 12, 8192) for w in files]
    torch.cuda.synchronize()
    got = []
    for i in range(40):
        w, method, layer = files[i & 1], GGUFLinearMethod(None), torch.nn.Module()
        method.create_weights(layer, 1024, [8192], 1024, 8192, torch.float16)
        for sid, part in ((None, w),) if i % 4 < 2 else ((0, w[:4096]), (1, w[4096:])):
            layer.weight.weight_loader(layer.weight, part.clone(), sid)
            layer.weight_type.weight_loader(layer.weight_type, torch.tensor(12), sid)
        method.process_weights_after_loading(layer)
        got.append(method.apply(layer, x))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i & 1]) for i, y in enumerate(got))


@pytest.mark.parametrize("types", [("Q4_K", "Q4_K", "Q6_K"), ("Q5_K", "Q5_K", "Q6_K"), ("Q3_K", "Q3_K", "Q5_K"), ("IQ3_S", "IQ3_S", "IQ4_XS"),
                                   ("IQ4_XS", "IQ4_XS", "Q5_K"), ("Q8_0", "Q4_1", "Q6_K")])
@pytest.mark.parametrize("K", [768, 2560, 3072, 3584, 5120])
def test_merged_shards_are_multiplied_where_they_lie(native_libs, types, K):
    """Whatever the hidden size, no shard is copied: `linear_runs` answers, and with what the shards' own products give."""
    from helpers import TYPES, rel_l2
    from vllm_gguf_plugin import native
    from vllm_gguf_plugin.quantization.linear import _fused_mul_mat_gguf

    ids = [TYPES[n] for n in types]
    method, layer, parts = merged_layer(ids, [264, 136, 72], K)
    for M in (1, 2, 3, 8, 17, 130):
        x = (torch.randn(M, K, device=DEV) / 8).half()
        y = native.linear_runs(x, layer.weight, layer.weight.gguf_runs)
        assert y is not None, (types, K, M)
        want = torch.cat([_fused_mul_mat_gguf(x, w, t) for t, w in zip(ids, parts)], dim=1)
        assert rel_l2(y.float().cpu(), want.float().cpu()) <= 3e-4, (types, K, M)    # (shared tiles add fp32 sums in another order)
        assert torch.equal(method.apply(layer, x), y)
    torch.cuda.synchronize()
    assert capi.last_status() == 0


# rows of the three shards: columns on and off 16-byte boundaries, a shard of one row
@pytest.mark.parametrize("rows", [[264, 136, 72], [33, 1, 30]])
@pytest.mark.parametrize("types", [("Q4_K", "Q4_K", "Q6_K"), ("IQ3_S", "IQ3_S", "IQ4_XS"), ("Q4_K", "Q4_K", "Q4_K")])
def test_compiled_layer_equals_the_eager_one(native_libs, types, rows):
    """One operator in the compiled graph, with the eager call's bits; fp32 activations and other batches as well."""
    from helpers import TYPES

    ids, graphs = [TYPES[n] for n in types], []
    method, layer, _ = merged_layer(ids, rows, 1024)

    def backend(gm, inputs):
        graphs.append([str(n.target) for n in gm.graph.nodes if n.op == "call_function"])
        return gm.forward

    torch._dynamo.reset()
    compiled = torch.compile(lambda x: method.apply(layer, x), backend=backend, fullgraph=True)
    for M, dtype in ((1, torch.float16), (2, torch.bfloat16), (9, torch.float16), (40, torch.float32)):
        if dtype == torch.float32 and types[0].startswith("IQ"):
            continue
        x = (torch.randn(M, 1024, device=DEV) / 8).to(dtype)
        assert torch.equal(compiled(x), method.apply(layer, x)), (M, dtype)
    assert graphs and all(g == ["_C_gguf.linear_runs"] or g == ["_C_gguf.linear_runs.default"] for g in graphs), graphs
    torch.cuda.synchronize()
    assert capi.last_status() == 0


def test_layer_copies_only_what_the_kernels_cannot_read_in_place(native_libs):
    """Rows a distance apart that Q4_K cannot be read at, and rows too long for the GEMV that takes a distance."""
    from helpers import TYPES, rel_l2

    op = torch.ops._C_gguf.linear_runs
    for K, names, pad in ((768, ("Q4_K", "Q6_K"), 6), (40960, ("Q4_K", "Q8_0"), 0)):
        ids = [TYPES[n] for n in names]
        parts = [weight(t, 24, K, seed=t) for t in ids]
        width = max(p.shape[1] for p in parts)
        buf = torch.zeros(48, width + pad, dtype=torch.uint8, device=DEV)
        W = buf[:, :width]
        runs = []
        for i, (t, p) in enumerate(zip(ids, parts)):
            W[24 * i:24 * i + 24, :p.shape[1]] = p
            runs += [t, 24 * i, 24, p.shape[1], 24]
        for M in (1, 2, 5, 30):
            x = (torch.randn(M, K, device=DEV) / 8).half()
            want = torch.cat([op(x, p, [t, 0, 24, p.shape[1], 24]) for t, p in zip(ids, parts)], dim=1)
            assert rel_l2(op(x, W, runs).float().cpu(), want.float().cpu()) <= 3e-4, (K, M)
    torch.cuda.synchronize()
    assert capi.last_status() == 0


def eager_cases():
    """(function of native.py, call through the public API, operator that the call becomes)"""
    from vllm_gguf_plugin import ops
    from vllm_gguf_plugin.quantization import fused_moe, vocal_embeds

    w, x = weight(12, 64, 256), torch.randn(20, 256, device=DEV).half()
    iq = weight(23, 64, 256)
    ids = torch.arange(4, device=DEV)
    w13, w2 = (torch.from_numpy(np.stack([synth.make_weight(2, 128, k, seed=e) for e in range(4)])).to(DEV) for k in (128, 64))
    tw, eid = torch.ones(3, 2, device=DEV), torch.zeros(3, 2, dtype=torch.int32, device=DEV)
    x3 = torch.randn(3, 128, device=DEV).half()
    method, layer, _ = merged_layer((12, 12, 14), [64, 32, 32], 256)
    one, plain, _ = merged_layer((12, 12, 12), [64, 32, 32], 256)
    return [("mul_mat", lambda: ops.ggml_mul_mat_vec_a8(w, x, 12, 64), "ggml_mul_mat_vec_a8"), ("mul_mat", lambda: ops.ggml_mul_mat_a8(w, x, 12, 64), "ggml_mul_mat_a8"),
            ("mul_mat", lambda: ops.ggml_dequant_matmul(iq, x, 23, 64), "dequant_matmul"),
            ("embed", lambda: vocal_embeds._apply_gguf_embedding(ids, w, 12, 256, torch.float16), "dequantize_rows"),
            ("moe", lambda: fused_moe._fused_moe_gguf(x3, w13, w2, tw, eid, 2, 2, "silu"), "fused_moe"),
            ("linear_runs", lambda: method.apply(layer, x), "linear_runs"), ("linear", lambda: one.apply(plain, x), "linear_runs")]


@pytest.mark.parametrize("i", range(7))
def test_dispatch_modes_and_compilation_see_the_operator(native_libs, monkeypatch, i):
    """The eager function serves the plain call; a dispatch mode, a traced and a compiled call see the registered operator and
    get the same bits."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from vllm_gguf_plugin import native

    name, call, op = eager_cases()[i]
    answers, function = [], getattr(native, name)

    def recorded(*args):
        answers.append(function(*args))
        return answers[-1]

    monkeypatch.setattr(native, name, recorded)
    want = call()
    assert len(answers) == 1 and answers[0] is not None
    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Mode():
        got = call()
    assert answers[-1] is None and f"_C_gguf.{op}.default" in seen, seen
    assert torch.equal(got, want)
    monkeypatch.setattr(native, name, function)
    graphs = []

    def backend(gm, inputs):
        graphs.append([str(n.target) for n in gm.graph.nodes if n.op == "call_function"])
        return gm.forward

    torch._dynamo.reset()
    assert torch.equal(torch.compile(call, backend=backend)(), want)
    assert any(op in t for g in graphs for t in g), graphs
