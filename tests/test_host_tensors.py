"""Operators that launch kernels on a tensor's address refuse tensors in host memory before anything is queued."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from hcomm_b200._stream import raw_stream
from hcomm_b200.ops.moe import MoeExchange


def test_no_stream_for_a_host_tensor():
    with pytest.raises(ValueError, match="CUDA"):
        raw_stream(torch.zeros(4))


def test_moe_exchange_refuses_host_tensors():
    class Library:
        def __getattr__(self, name):
            raise AssertionError(f"{name} was called with a host address")
    moe = MoeExchange.__new__(MoeExchange)
    moe.comm, moe.num_experts, moe.topk, moe.hidden, moe.max_tokens = SimpleNamespace(size=1), 8, 2, 512, 4
    moe._lib, moe._h = Library(), ctypes.c_void_p()
    x = torch.zeros(4, 512, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="CUDA"):
        moe.dispatch(x, torch.zeros(4, 2, dtype=torch.int32))
    with pytest.raises(ValueError, match="CUDA"):
        moe.combine(torch.zeros(8, 512, dtype=torch.bfloat16), torch.zeros(4, 2))
