"""Options of the plain GEMM that are read from the environment at its first call: each runs in a process of its own."""
import os
import subprocess
import sys
from pathlib import Path

import pytest


def run(program, **env):
    root = Path(__file__).resolve().parent.parent
    res = subprocess.run([sys.executable, "-c", program], capture_output=True, text=True, timeout=240, cwd=root, env=dict(os.environ, PYTHONPATH=str(root), **env))
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-3000:]
    return res.stdout


def test_wide_tiles_can_be_switched_off():
    program = """
import ctypes
from hcomm_b200 import _lib
lib = _lib.load()
bn, caps = ctypes.c_int(), (ctypes.c_int * 4)(74, 33, 22, 15)
print(lib.HcommToolGemmTileOf(8192, 28672, 8192, caps, ctypes.byref(bn), None), bn.value)
"""
    assert run(program, HCOMM_GEMM_WIDE="1").split() == ["1", "512"]
    kernel, width = run(program, HCOMM_GEMM_WIDE="0").split()
    assert kernel != "1" and int(width) <= 256


@pytest.mark.gpu
def test_a_large_shape_is_measured_at_its_first_use():
    out = run("""
import ctypes, torch
from hcomm_b200 import _lib
from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
lib = _lib.load()

def tuned(m, n, k):
    bn, group = ctypes.c_int(-1), ctypes.c_int(-1)
    lib.HcommGemmGetTuned(m, n, k, ctypes.byref(bn), ctypes.byref(group))
    return bn.value, group.value

for m, n, k in [(2048, 8192, 8192), (777, 14336, 10240), (256, 512, 512)]:
    a = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    b = (torch.randn(n, k, device="cuda") * 0.02).to(torch.bfloat16)
    assert tuned(m, n, k) == (0, 0)
    out = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    graph = torch.cuda.CUDAGraph()
    lib.HcommGemmSetTuning(0, 256)          # a forced width is not measured; it also loads the kernels ahead of the capture
    gemm_bf16(a, b, out)
    lib.HcommGemmSetTuning(0, 0)
    with torch.cuda.graph(graph):           # nor is a stream that is being captured
        gemm_bf16(a, b, out)
    assert tuned(m, n, k) == (0, 0)
    got = gemm_bf16(a, b)
    bn, group = tuned(m, n, k)
    large = 2 * m * n * k >= 2e11
    assert (32 <= bn <= 512 and 2 <= group <= 32) if large else (bn, group) == (0, 0), (bn, group)
    again = gemm_bf16(a, b)
    graph.replay()
    torch.cuda.synchronize()
    assert take_kernel_error() == 0 and tuned(m, n, k) == (bn, group) and torch.equal(got, again)
    ref = a.float() @ b.float().t()
    for c in (got, out):
        assert (c.float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item()
print("ok")
""", HCOMM_GEMM_AUTOTUNE="1")
    assert "ok" in out
