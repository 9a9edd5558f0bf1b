"""The short way from Python to the C entry points: taken for plain CUDA tensors, left to the general way for anything else."""
import subprocess
import sys
import sysconfig
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_the_interpreter_lock_is_held_again_behind_an_exception(tmp_path):
    # an allocation that fails inside an entry point comes out of it as a C++ exception, of which a Python error is made
    so = tmp_path / "released_probe.so"
    cmd = ["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{sysconfig.get_paths()['include']}", str(ROOT / "tests" / "released_probe.cc"), "-o", str(so)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    program = "import released_probe as p; print(*p.returns(), p.throws(), *p.returns())"
    res = subprocess.run([sys.executable, "-c", program], capture_output=True, text=True, timeout=60, cwd=tmp_path)
    assert res.returncode == 0 and res.stdout.split() == ["0", "1", "1", "0", "1"], res.stdout + res.stderr


def test_threads_that_come_at_once_get_one_extension():
    # ranks may be threads of one process, and any operator may be the first call
    program = """
import sys, threading, time
import torch.distributed
from hcomm_b200 import _ext, _lib
if not _ext._PATH.exists():
    _ext.extension()
    _ext._MODULE = None
load = _lib.load
_lib.load = lambda: (time.sleep(0.2), load())[1]        # all of them are between the first look and the load
torch.cuda.is_available = lambda: True
found = []
threads = [threading.Thread(target=lambda f=f: found.append(f())) for f in [_ext.extension, _ext.native_calls] * 4]
for t in threads:
    t.start()
for t in threads:
    t.join()
print(len(found), len({id(m) for m in found}), found[0] is sys.modules["_hcomm_torch"], _ext.native_calls() is found[0])
"""
    res = subprocess.run([sys.executable, "-c", program], capture_output=True, text=True, timeout=240, cwd=ROOT)
    assert res.returncode == 0 and res.stdout.split() == ["8", "1", "True", "True"], res.stdout + res.stderr


def test_an_extension_that_does_not_load_is_said_once(monkeypatch, tmp_path):
    import warnings

    import torch

    from hcomm_b200 import _ext

    def fails():
        raise ImportError("undefined symbol")
    (tmp_path / "ext.so").touch()
    monkeypatch.setattr(_ext, "_CALLS", False)
    monkeypatch.setattr(_ext, "_PATH", tmp_path / "ext.so")
    monkeypatch.setattr(_ext, "extension", fails)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.delenv("HCOMM_LIBRARY", raising=False)
    with pytest.warns(UserWarning, match="undefined symbol"):
        assert _ext.native_calls() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _ext.native_calls() is None


def test_without_a_gpu_the_general_way_is_taken():
    import torch

    from hcomm_b200 import _ext
    if torch.cuda.is_available():
        pytest.skip("this machine has a GPU")
    assert _ext.native_calls() is None
    assert _ext.Short("gemm_bf16", "HcommGemmBf16")(None, None, None) is None


@pytest.mark.gpu
def test_plain_tensors_go_the_short_way_and_others_do_not():
    import torch
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    from hcomm_b200 import _ext
    from hcomm_b200.ops.gemm import gemm_bf16
    torch.cuda.set_device(0)
    calls, entry = _ext.native_calls(), _ext.entry("HcommGemmBf16")
    assert calls is not None
    a = torch.randn(40, 72, device="cuda").to(torch.bfloat16)
    b = torch.randn(24, 72, device="cuda").to(torch.bfloat16)
    want = gemm_bf16(a, b)

    def short(*args):
        return calls.gemm_bf16(entry, *args)
    assert torch.equal(short(a, b, None), want)
    out = torch.empty_like(want)
    assert short(a, b, out) is out and torch.equal(out, want)
    assert torch.equal(short(a[::2], b, None), want[::2])                     # a longer pitch
    p = torch.nn.Parameter(b)
    assert torch.equal(short(a, p, None), want) and not short(a, p, None).requires_grad
    with torch.autocast("cuda"), torch.inference_mode():
        assert torch.equal(short(a, b, None), want)

    class Sub(torch.Tensor):
        pass
    for args in ((a.float(), b, None), (a.cpu(), b, None), (a, b.t(), None), (a.t().contiguous().t(), b, None), (a[0], b, None), (a.as_subclass(Sub), b, None),
                 (a, b[:, :64], None), (a, b.cpu(), None), (1, b, None), (a, b, out.cpu()), (a, b, 5)):
        assert short(*args) is None

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    for mode in (Function, Dispatch):
        with mode():
            assert short(a, b, None) is None
            got = gemm_bf16(a, b)
        assert torch.equal(got, want)
    seen = []
    torch.vmap(lambda v: seen.append(short(v, b, None)) or v)(torch.stack([a, a]))
    assert seen == [None]
    for bad, error in (((a.float(), b), TypeError), ((a, b[:, :64]), ValueError), ((a.cpu(), b), RuntimeError), ((a, b.t()), ValueError)):
        with pytest.raises(error):
            gemm_bf16(*bad)
    with pytest.raises(Exception, match="HCCL_E_PARA"):
        gemm_bf16(a[:, :70].contiguous(), b[:, :70].contiguous())             # the kernel wants K in multiples of 8


@pytest.mark.gpu
def test_operators_and_exchange_by_both_ways():
    import torch

    import hcomm_b200 as hb
    from hcomm_b200.ops.moe import MoeExchange
    torch.cuda.set_device(0)
    comm = hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=4)
    moe = MoeExchange(comm, 8, 2, 512, 16, capacity_factor=1.0)
    try:
        x = torch.randn(1000, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        for name in ("all_reduce", "all_reduce_scaled", "reduce_scatter", "all_gather", "all_to_all"):
            out, other = torch.empty_like(x), torch.empty_like(x)
            extra = {"scale": 0.5} if name == "all_reduce_scaled" else {}
            assert comm._short(name, x, torch.empty_like(x), None, 0, 1.0)
            assert not comm._short(name, x, out, stream) and not comm._short(name, x[::2], out[::2], None) and not comm._short(name, x, out.cpu(), None)
            assert getattr(comm, name)(x, out, **extra) is out
            getattr(comm, name)(x, other, stream=stream, **extra)
            assert torch.equal(out, other) and torch.equal(out, x * 0.5 if extra else x)
        with pytest.raises(KeyError):
            comm.all_reduce(x, op="mean")
        with pytest.raises(ValueError):
            comm.all_gather(x[::2], x[::2])
        t = torch.randn(16, 512, device="cuda").to(torch.bfloat16)
        idx = torch.randint(0, 8, (16, 2), device="cuda", dtype=torch.int32)
        idx[:, 1] = (idx[:, 0] + 1) % 8
        gates = torch.rand(16, 2, device="cuda")
        rec = moe.dispatch(t, idx)
        assert rec.num_rows == 32
        y = rec.dequantized(32).to(torch.bfloat16)
        out = torch.empty(16, 512, device="cuda", dtype=torch.bfloat16)
        got = moe.combine(y, gates)
        assert moe.combine(y, gates, out) is out and torch.equal(out, got)
        for bad in ((t.float(), idx), (t, idx.long()), (t[:, :256], idx), (t, idx[:8])):
            with pytest.raises(AssertionError):
                moe.dispatch(*bad)
        with pytest.raises(AssertionError):
            moe.combine(y.float(), gates)
    finally:
        moe.destroy()
    with pytest.raises(Exception):
        moe.dispatch(t, idx)
    comm.destroy()
