"""Setting up an MoE exchange when its device memory cannot be had, with stand-ins for the CUDA allocator."""
import ctypes

import pytest

from hcomm_b200 import _lib

HCCL_E_MEMORY, HCCL_E_RUNTIME = 3, 15


def make(failing, experts=256, tokens=4096, topk=8):
    left, overflow, rows = ctypes.c_int(-1), ctypes.c_uint64(), ctypes.c_uint64()
    rc = _lib.load().HcommToolMoeScratch(experts, tokens, topk, failing, ctypes.byref(left), ctypes.byref(overflow), ctypes.byref(rows))
    return rc, left.value, overflow.value, rows.value


@pytest.mark.parametrize("failing,code", [(1, HCCL_E_MEMORY), (2, HCCL_E_RUNTIME)])
def test_a_block_that_cannot_be_had_is_an_error_and_nothing_is_kept(failing, code):
    rc, left, _, _ = make(failing)
    assert rc == code and left == 0


def test_parts_of_the_block_do_not_overlap():
    rc, left, overflow, rows = make(0, experts=64)
    assert rc == 0 and left == 1 and overflow >= 64 and rows >= overflow + 2
