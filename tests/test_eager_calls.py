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
