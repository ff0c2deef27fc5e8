"""CPU: the C-ABI library builds, loads, exports every declared symbol and validates arguments
(no kernel is launched here)."""
import ctypes
import re

import pytest

from helpers import ROOT


def declared_symbols():
    text = (ROOT / "include" / "gguf_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(gguf_b200_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(native_libs):
    lib = ctypes.CDLL(str(native_libs[0]))
    names = declared_symbols()
    assert len(names) >= 15
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/gguf_b200.h but not exported"


def test_binding_table_covers_the_header(native_libs):
    from gguf_b200 import capi

    assert set(declared_symbols()) == set(capi.SIGNATURES)


def test_geometry_and_error_codes(native_libs):
    from gguf_b200 import capi

    lib = capi.lib()
    sizes = {2: (32, 18), 8: (32, 34), 12: (256, 144), 14: (256, 210), 16: (256, 66), 23: (256, 136)}
    for t, (bs, ts) in sizes.items():
        assert lib.gguf_b200_block_size(t) == bs and lib.gguf_b200_type_size(t) == ts
    assert lib.gguf_b200_type_size(10) == 84 and lib.gguf_b200_block_size(11) == 256
    assert lib.gguf_b200_type_size(9) == 0 and lib.gguf_b200_block_size(9) == 0
    assert lib.gguf_b200_q8_1_row_bytes(1024) == 1024 // 32 * 36
    assert lib.gguf_b200_q8_1_row_bytes(800) == 1024 // 32 * 36
    assert lib.gguf_b200_moe_block_size(2) == 64 and lib.gguf_b200_moe_block_size(11) == 64 and lib.gguf_b200_moe_block_size(16) == 0
    assert lib.gguf_b200_workspace_bytes(capi.OP_GEMV, 12, 2, 0, 4096) == 2 * 4096 + 2 * 128 * 8
    assert lib.gguf_b200_workspace_bytes(capi.OP_MMQ, 8, 4, 0, 1024) == 4 * 1024 * 2
    assert lib.gguf_b200_workspace_bytes(capi.OP_MMQ, 12, 4, 0, 1024) == 4 * (1024 + 64) * 2
    # argument validation happens before any CUDA call
    null = ctypes.c_void_p(0)
    p = ctypes.c_void_p(4096)
    assert lib.gguf_b200_mul_mat_vec_a8(p, p, p, p, 1 << 20, 9, 1, 1, 8, 256, null) == -1   # type (Q8_1 is not a weight type)
    assert lib.gguf_b200_mul_mat_a8(p, p, p, p, 1 << 20, 21, 1, 1, 8, 256, null) == -1       # IQ3_S has no tiled kernel
    assert lib.gguf_b200_mul_mat_vec_a8(p, p, p, p, 1 << 20, 12, 7, 1, 8, 256, null) == -2  # dtype
    assert lib.gguf_b200_mul_mat_vec_a8(p, p, p, p, 1 << 20, 12, 1, 1, 8, 100, null) == -3  # K % 256
    assert lib.gguf_b200_mul_mat_vec_a8(null, p, p, p, 1 << 20, 12, 1, 1, 8, 256, null) == -4
    assert lib.gguf_b200_mul_mat_vec_a8(ctypes.c_void_p(4100), p, p, p, 1 << 20, 12, 1, 1, 8, 256, null) == -4  # alignment
    assert lib.gguf_b200_mul_mat_vec_a8(p, p, p, p, 16, 12, 1, 1, 8, 256, null) == -5       # workspace
    assert lib.gguf_b200_mul_mat_a8(p, p, p, p, 1 << 20, 16, 1, 1, 8, 256, null) == -1      # IQ has no q8_1 GEMM
    assert lib.gguf_b200_dequant_matmul(p, p, p, p, 0, 12, 1, 1, 8, 256, null) == -1
    assert lib.gguf_b200_dequant_matmul(p, p, p, p, 0, 16, 0, 1, 8, 256, null) == -2        # fp32 not fused
    assert lib.gguf_b200_dequantize(p, 12, p, 1, 100, null) == -3
    assert lib.gguf_b200_mul_mat_vec_a8(p, p, p, p, 0, 12, 1, 0, 8, 256, null) == 0          # empty batch
    assert b"workspace" in lib.gguf_b200_error_string(-5)
    # dense GEMM workspace: activations, and the parts of tiles that several CTAs share: two tiles of 128 rows for each of up to
    # 148 CTAs, in fp32, behind a counter per tile
    act = lambda m, k: (m * (k + (k // 32 + 63) // 64 * 64) * 2 + 255) // 256 * 256
    for op, t, m, n, k, shared in ((capi.OP_MMQ, 12, 512, 14336, 4096, None), (capi.OP_MMQ, 12, 512, 4096, 14336, True), (capi.OP_MMQ, 12, 64, 4096, 14336, True),
                                   (capi.OP_MMQ, 12, 512, 18944, 4096, None), (capi.OP_DEQUANT_MATMUL, 16, 128, 1024, 28672, True),
                                   (capi.OP_DEQUANT_MATMUL, 16, 128, 128 * 148, 4096, False), (capi.OP_DEQUANT_MATMUL, 16, 128, 8192, 28672, True)):
        room = lib.gguf_b200_workspace_bytes(op, t, m, n, k) - (act(m, k) if op == capi.OP_MMQ else 0)
        assert 0 <= room <= 2 * 148 * 128 * 384 * 4 + (1 << 20) and room % 256 == 0
        assert shared is None or (room > 0) == shared, (op, t, m, n, k, room)
        assert lib.gguf_b200_scratch_bytes(op, t, m, n, k) == room + (act(m, k) if op == capi.OP_MMQ else 0)   # nothing allocated that no call uses
    # a few tokens: what the small-batch kernel needs, and not also what the tiled one would
    assert lib.gguf_b200_workspace_bytes(capi.OP_GEMV, 12, 8, 4096, 14336) < lib.gguf_b200_scratch_bytes(capi.OP_GEMV, 12, 8, 4096, 14336)
    assert lib.gguf_b200_scratch_bytes(capi.OP_MMQ, 14, 8, 4096, 14336) == lib.gguf_b200_scratch_bytes(capi.OP_GEMV, 14, 8, 4096, 14336)


def test_tensor_parallel_entry_points_validate_arguments(native_libs):
    from gguf_b200 import capi

    lib = capi.lib()
    null = ctypes.c_void_p(0)
    p = ctypes.c_void_p(4096)
    two = (ctypes.c_void_p * 2)(4096, 8192)
    ptrs = ctypes.cast(two, ctypes.c_void_p)
    # decode: W, X, packet arenas, epochs, slot, add_slot, add_scale, add_parts, slot_packets, ws, ws_bytes, type, dtype, N_local, K, rank, world, stream
    args = lambda **kw: [kw.get("W", p), kw.get("X", p), kw.get("y", ptrs), kw.get("e", p), kw.get("slot", 0), kw.get("add", -1), 0.0,
                         kw.get("parts", 1), kw.get("sp", 1024), p, 1 << 20, kw.get("type", 12), 1, 64, 256, kw.get("rank", 0),
                         kw.get("world", 2), null]
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(y=null)) == -4
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(e=null)) == -4
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(X=null)) == -4          # no activations at all
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(world=9)) == -3
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(rank=2)) == -3
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(slot=-1)) == -3
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(sp=100)) == -3          # slot too small for world * N_local
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(add=0)) == -3           # a call cannot consume its own slot
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(type=9)) == -1
    assert lib.gguf_b200_mul_mat_vec_a8_tp(*args(add=1, parts=3)) == -3  # partial vectors come one per rank, or not at all
    # row-parallel: same arguments, N and K_local in place of N_local and K; a slot holds world * N fp32 partials
    assert lib.gguf_b200_mul_mat_vec_a8_tp_rowpar(*args(y=null)) == -4
    assert lib.gguf_b200_mul_mat_vec_a8_tp_rowpar(*args(world=9)) == -3
    assert lib.gguf_b200_mul_mat_vec_a8_tp_rowpar(*args(sp=200)) == -3   # 2 ranks x 64 rows x 8 bytes > 200 x 4
    assert lib.gguf_b200_mul_mat_vec_a8_tp_rowpar(*args(type=9)) == -1
    assert lib.gguf_b200_tp_unpack_sum(null, p, 0, 1024, 64, 2, p, 1, null) == -4
    assert lib.gguf_b200_tp_unpack_sum(p, p, 0, 1024, 64, 9, p, 1, null) == -3
    assert lib.gguf_b200_tp_unpack_sum(p, p, 0, 1024, 4096, 2, p, 1, null) == -3   # partials beyond the slot
    assert lib.gguf_b200_tp_unpack(null, p, 0, 1, 1024, 64, p, 64, 1, null) == -4
    assert lib.gguf_b200_tp_unpack(p, p, 0, 1, 1024, 2048, p, 2048, 1, null) == -3   # n beyond the slot
    assert lib.gguf_b200_tp_unpack(p, p, 0, 1, 1024, 64, p, 64, 9, null) == -2
    # prefill: op, W, X, outputs, flags, epochs, slot, ws, ws_bytes, type, dtype, M, N_local, K, rank, world, stream
    margs = lambda **kw: [kw.get("op", capi.OP_MMQ), p, p, kw.get("y", ptrs), ptrs, p, 0, p, 1 << 30, kw.get("type", 12),
                          kw.get("dtype", 1), 32, 64, 256, 0, kw.get("world", 2), null]
    assert lib.gguf_b200_matmul_tp(*margs(y=null)) == -4
    assert lib.gguf_b200_matmul_tp(*margs(op=capi.OP_GEMV)) == -3
    assert lib.gguf_b200_matmul_tp(*margs(world=0)) == -3
    assert lib.gguf_b200_matmul_tp(*margs(type=16)) == -1                # IQ types go through OP_DEQUANT_MATMUL
    assert lib.gguf_b200_matmul_tp(*margs(op=capi.OP_DEQUANT_MATMUL, type=12)) == -1
    assert lib.gguf_b200_matmul_tp(*margs(op=capi.OP_DEQUANT_MATMUL, type=16, dtype=0)) == -2
    assert lib.gguf_b200_tp_wait(null, p, 0, 2, null) == -4
    assert lib.gguf_b200_tp_wait(p, p, 0, 0, null) == -3
    lib.gguf_b200_set_wait_limit_cycles(0)                                # restores the default; no device call


def test_ops_module_fails_loudly_without_extension(tmp_path, monkeypatch):
    """The product path has no fallback: importing ops next to a missing extension raises."""
    import importlib
    import shutil
    import sys

    pkg = tmp_path / "vllm_gguf_plugin"
    pkg.mkdir()
    src = ROOT / "vllm-gguf-plugin-prism_b200" / "vllm_gguf_plugin"
    shutil.copy(src / "ops.py", pkg / "ops.py")
    (pkg / "__init__.py").write_text("")
    saved = {k: sys.modules.pop(k) for k in list(sys.modules) if k.split(".")[0] == "vllm_gguf_plugin"}
    monkeypatch.syspath_prepend(str(tmp_path))
    try:
        try:
            importlib.import_module("vllm_gguf_plugin.ops")
            raised = False
        except ImportError as e:
            raised = "not built" in str(e)
        assert raised
    finally:
        for k in [k for k in sys.modules if k.split(".")[0] == "vllm_gguf_plugin"]:
            del sys.modules[k]
        sys.modules.update(saved)


def test_quantizers_let_the_product_start_only_behind_their_own_wait():
    """A product reads weights as soon as it starts, so the quantizer ahead of it must not release it (pdl_trigger) before the
    work ahead of the call -- a kernel that wrote those weights, for one -- is complete (pdl_wait)."""
    src = (ROOT / "vllm-gguf-plugin-prism_b200" / "csrc" / "quantize_q8_1.cu").read_text()
    kernels = re.split(r"^__global__", src, flags=re.M)[1:]
    assert len(kernels) == 3
    for k in kernels:
        k = k.replace("if (tp.early) pdl_trigger();", "")      # (the caller's weights are known to be complete)
        assert 0 < k.index("pdl_wait();") < k.index("pdl_trigger();")
    assert src.count("if (tp.early) pdl_trigger();") == 1


def test_tiles_are_shared_where_that_pays(native_libs):
    """The plan of the tiled kernel shows in the room it asks for: 112 row tiles on 148 SMs are not worth cutting into runs for a
    few tokens (Q5_K, 24 tokens: 28.3 us in runs, 25.5 whole), 32 row tiles of long rows are."""
    from gguf_b200 import capi

    lib = capi.lib()
    for t in (2, 8, 10, 12, 13):
        for m in (17, 24, 32, 64):
            n, k = 14336, 4096
            columns = k + (k // 32 + 63) // 64 * 64 if t in (2, 12, 13) else k
            assert lib.gguf_b200_workspace_bytes(capi.OP_MMQ, t, m, n, k) == (m * columns * 2 + 255) // 256 * 256, (t, m)
            assert lib.gguf_b200_workspace_bytes(capi.OP_MMQ, t, m, 4096, 14336) > 1 << 20


@pytest.mark.parametrize("t,m,n,k,tile", [(8, 272, 8192, 28672, 288), (8, 300, 8192, 28672, 320), (2, 300, 8192, 28672, 320), (3, 352, 8192, 28672, 352),
                                          (21, 700, 8192, 28672, 352), (8, 700, 28672, 8192, 352)])
def test_tiles_beyond_256_tokens_where_they_pay(native_libs, t, m, n, k, tile):
    """Tiles of 257 to 384 tokens take less time than two or three smaller ones in these calls (8192x28672: Q8_0, 272 tokens 135 us in one tile, 155 in
    two; 300 tokens 137 and 157; Q4_0 135 and 147; Q4_1, 352 tokens 154 and 162; IQ3_S, 700 tokens 251 in two and 263 in three)."""
    from gguf_b200 import capi

    op = capi.OP_DEQUANT_MATMUL if t == 21 else capi.OP_MMQ
    columns = k + ((k // 32 + 63) // 64 * 64 if t in (2, 3) else 0)
    activations = 0 if t == 21 else (m * columns * 2 + 255) // 256 * 256
    tiles = (n // 128) * ((m + tile - 1) // tile)
    counters = (tiles * 4 + 255) // 256 * 256
    # runs over all SMs: two parts of 128 rows by a tile's tokens for each of 148 CTAs
    assert capi.lib().gguf_b200_workspace_bytes(op, t, m, n, k) == activations + counters + 2 * 148 * 128 * tile * 4


def test_moe_products_read_their_work_list_past_l1():
    """The products of a MoE step read the work list ahead of their own griddepcontrol.wait: only loads that do not take the L1's word may do that,
    since the list lies at the same addresses in every step.  Plain loads of it, and of the routing, stand behind the wait."""
    csrc = ROOT / "vllm-gguf-plugin-prism_b200" / "csrc"
    plain = r"p\.(?:passes|sorted|row_scale)\[|(?<![\w*] )\*p\.n_passes\b|__ldg\(p\.(?:sorted|row_scale)\b"
    mmq = (csrc / "mmq_kernel.cuh").read_text()
    at = mmq.index("waited ? p.passes[q.outer] : ld_older(p.passes + q.outer)")
    epilogue = mmq.index("pdl_wait();", mmq.index("auto epilogue = "))
    for m in re.finditer(plain, mmq):
        assert m.start() == at + len("waited ? ") or m.start() > epilogue, m.group()
    assert mmq[epilogue:].index("mmq_tile(p, e, true)") < 60                     # the epilogue's tile: right behind its wait
    calls = [m.start() for m in re.finditer(r"mmq_tile\(p, q, (?:true|waited)\)", mmq)]
    assert len(calls) == 2                                                        # the decoders' and the activation loader's
    for c in calls:
        assert 0 < c - mmq.rindex("pdl_wait();", 0, c) < 250
    small = (csrc / "smallm.cuh").read_text()
    producer, consumers = small.index("if (producer) {"), small.index("  pdl_wait();\n  for (; u < u1; ++tile)")
    for m in re.finditer(plain, small):
        before = small[m.start() - len("waited ? "):m.start()]
        assert before == "waited ? " or m.start() > consumers or "auto outputs" in small[producer:m.start()], m.group()
    assert small.count("ld_older(p.n_passes)") == 1 and mmq.count("ld_older(p.n_passes)") == 1
    assert (csrc / "common.cuh").read_text().count("ld.relaxed.gpu.global") == 2
