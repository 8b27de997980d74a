"""The compiled call path (awesome-cute_b200/csrc/w4a16_torch.cpp) and what happens beside it: without the module, with an
error of the library, on layers whose tensors are not plain buffers."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

import __graft_entry__ as entry

pkg = entry.load_package()
from awesome_cute_b200 import _lib  # noqa: E402

WITHOUT = r"""
import sys, warnings
sys.modules['awesome_cute_b200._torch_calls'] = None        # as if it were not built, or for another torch
import torch
import __graft_entry__ as entry
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter('always')
    pkg = entry.load_package()
assert any('_torch_calls' in str(w.message) for w in seen), seen
A, C = torch.zeros((16, 256), dtype=torch.half), torch.zeros((16, 256), dtype=torch.half)
B, s = torch.zeros((16, 512), dtype=torch.int), torch.zeros((2, 256), dtype=torch.half)
try:
    pkg.mul(A, B, C, s, torch.zeros(32, dtype=torch.int))
except RuntimeError as e:
    assert 'no CPU implementation' in str(e), e
layer = pkg.Layer(256, 256, 128)
if torch.cuda.is_available():
    layer = layer.cuda()
    w, sc = torch.randn(256, 256).half().cuda(), torch.full((2, 256), 0.01).half().cuda()
    layer.B, layer.s = pkg.quantize_pack_device(w, sc, 128)
    x = torch.randn(3, 256).half().cuda()
    y = torch.zeros(3, 256).half().cuda()
    pkg.mul(x, layer.B, y, layer.s, layer.workspace)
    assert torch.equal(layer(x), y) and bool(y.any())
print('ok')
"""


def run_without():
    r = subprocess.run([sys.executable, "-c", WITHOUT], cwd=entry.ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-1000:] + r.stderr[-2000:]


def test_the_package_works_without_the_module():
    run_without()


@pytest.mark.gpu
def test_the_package_works_without_the_module_on_a_gpu():
    run_without()


def operands(m=4, n=256, k=256):
    dev = "cuda:0"
    return (torch.randn((m, k), device=dev).half(), torch.zeros((k // 16, 2 * n), dtype=torch.int, device=dev),
            torch.zeros((m, n), dtype=torch.half, device=dev), torch.full((k // 128, n), 0.01, dtype=torch.half, device=dev),
            torch.zeros(n // 128 * 16, dtype=torch.int, device=dev))


@pytest.mark.gpu
def test_an_error_of_the_library_is_raised_and_the_call_not_repeated():
    calls = []
    gemm = ctypes.CFUNCTYPE(ctypes.c_int, *_lib._GEMM_ARGS)(lambda *a: calls.append("gemm") or _lib.ERR_CUDA)
    pack = ctypes.CFUNCTYPE(ctypes.c_int, *_lib.SYMBOLS["w4a16_quantize_pack_device"][1])(lambda *a: calls.append("pack") or _lib.ERR_CUDA)
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value
    A, B, C, s, ws = operands()
    layer = pkg.Layer(256, 256, 128).cuda()
    w = torch.zeros((256, 256), dtype=torch.half, device="cuda:0")
    _lib.calls.bind(address(gemm), address(pack))
    try:
        with pytest.raises(RuntimeError, match="code 3"):
            pkg.mul(A, B, C, s, ws)
        with pytest.raises(RuntimeError, match="code 3"):
            layer(A)
        with pytest.raises(ValueError, match="code 3"):
            pkg.quantize_pack_device(w, s, 128)
    finally:
        _lib.calls.bind(address(_lib.lib.w4a16_marlin_gemm), address(_lib.lib.w4a16_quantize_pack_device))
    assert calls == ["gemm", "gemm", "pack"]
    pkg.mul(A, B, C, s, ws)
    torch.cuda.synchronize()
    assert bool(C.any())


@pytest.mark.gpu
def test_a_layer_whose_weights_are_no_buffer():
    A, B, C, s, ws = operands()
    layer = pkg.Layer(256, 256, 128).cuda()
    layer.s.copy_(s)
    del layer.B
    object.__setattr__(layer, "B", B)
    pkg.mul(A, B, C, s, ws)
    assert torch.equal(layer(A), C)
