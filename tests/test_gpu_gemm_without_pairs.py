"""The plain GEMM without CTA pairs (HCOMM_GEMM_PAIR=0, or a device that cannot hold a cluster): both of its tile widths, at
the edges of tiles and of K.  The variable is read at the first call, so a process of its own runs each case."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import torch
from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
for m, n, k in [(1, 8, 8), (127, 136, 72), (128, 256, 64), (129, 264, 520), (300, 2048, 1032), (2000, 128, 256), (700, 4104, 64)]:
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    b = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    full = torch.full((m, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm_bf16(a, b, full[:, :n])
    torch.cuda.synchronize()
    assert take_kernel_error() == 0 and bool((full[:, n:] == 7.0).all()), (m, n, k)
    ref = a.double() @ b.double().t()
    # one rounding to bf16 (half a step, 2^-9) and fp32 sums of k products (k * 2^-24 of the sum of magnitudes)
    bound = 2.0 ** -8 * ref.abs() + k * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t())
    assert bool(((full[:, :n].double() - ref).abs() <= bound).all()), (m, n, k)
print("ok")
"""


def test_gemm_without_pairs():
    root = Path(__file__).resolve().parent.parent
    res = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=240, cwd=root,
                         env=dict(os.environ, HCOMM_GEMM_PAIR="0", PYTHONPATH=str(root)))
    assert res.returncode == 0 and "ok" in res.stdout, res.stdout[-2000:] + res.stderr[-3000:]
