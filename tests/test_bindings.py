"""CPU: what the two binding libraries are tied to, and what happens where the narrower one cannot load."""
import shutil
import subprocess
import sys

import pytest

from conftest import PKG


def undefined(so):
    out = subprocess.run(["nm", "-D", "--undefined-only", str(so)], check=True, capture_output=True, text=True).stdout
    return {line.split()[-1].split("@")[0] for line in out.splitlines()}


@pytest.mark.skipif(shutil.which("nm") is None, reason="needs binutils")
def test_operator_library_needs_only_the_stable_interfaces(native_libs):
    """`_C_gguf.abi3.so` keeps what its name says: torch's C shim, Python's limited API, no C++ symbol of torch."""
    names = undefined(native_libs[1])
    assert any(n.startswith("aoti_torch_") for n in names)
    assert not [n for n in names if n.startswith(("_ZN2at", "_ZN3c10", "_ZN5torch", "_ZNK2at", "_ZNK3c10", "_ZNK5torch", "THP"))]
    assert {n for n in names if n.startswith(("Py", "_Py"))} <= {"PyModule_Create2"}


def run(code):
    return subprocess.run([sys.executable, "-c", f"import sys; sys.path.insert(0, {str(PKG)!r})\n{code}"], capture_output=True, text=True, timeout=300)


def test_calls_go_through_the_operators_without_the_eager_module(native_libs):
    r = run("sys.modules['vllm_gguf_plugin._eager'] = None\n"
            "import torch\nfrom vllm_gguf_plugin import native, ops\n"
            "from vllm_gguf_plugin.quantization import GGUFLinearMethod\n"
            "assert native.linear(None, None, 0) is None and native.moe() is None\n"
            "x = torch.zeros(2, 256, device='meta', dtype=torch.float16)\n"
            "assert ops.ggml_mul_mat_a8(torch.zeros(8, 144, dtype=torch.uint8, device='meta'), x, 12, 8).shape == (2, 8)\n")
    assert r.returncode == 0, r.stderr
    assert "operator dispatcher" in r.stderr


def test_eager_module_refuses_another_torch(native_libs):
    r = run("import torch\ntorch.__version__ = '9.9.9'\n"
            "try:\n    from vllm_gguf_plugin import _eager\nexcept ImportError as e:\n    print('refused:', e)\n")
    assert "refused: built for torch" in r.stdout, r.stdout + r.stderr
