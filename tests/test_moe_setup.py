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


def test_launch_of_a_single_ranks_dispatch():
    def shape(tokens, topk, experts, hidden, ctas=296, sms=148):
        out = (ctypes.c_int * 3)()
        _lib.load().HcommToolMoeDispatchShape(tokens, topk, experts, hidden, ctas, sms, out)
        return tuple(out)
    alone, pairs = (296, 512, 1), (148, 1024, 2)
    # by the choices that have to be counted, sooner where rows are small
    assert shape(2125, 8, 256, 512) == alone and shape(2126, 8, 256, 512) == pairs
    assert shape(2048, 8, 256, 4096) == shape(3000, 8, 256, 4096) == alone and shape(3001, 8, 256, 4096) == pairs
    # by what has to be moved
    assert shape(6713, 1, 8, 8192) == alone and shape(6714, 1, 8, 8192) == pairs
    # two experts to a thread, but for many choices of small rows
    assert shape(1750, 8, 1024, 4096) == shape(1124, 8, 1024, 512) == alone and shape(1126, 8, 1024, 512) == (148, 1024, 1)
    assert shape(9000, 16, 1024, 512) == pairs
    # however few CTAs it may have
    assert shape(1, 8, 256, 7168, ctas=1) == (1, 512, 1)
    assert shape(4096, 8, 256, 7168, ctas=1) == (1, 1024, 1) and shape(4096, 8, 256, 7168, ctas=3) == (2, 1024, 2)
    for tokens in (1, 100, 3000, 100000):
        for experts in (8, 512, 513, 1024):
            ctas, threads, cluster = shape(tokens, 8, experts, 1024, ctas=min(296, tokens))
            assert 1 <= ctas <= min(296, tokens) and ctas % cluster == 0 and threads in (512, 1024) and ctas * threads <= 148 * 1024
            assert cluster == 1 or threads == 1024
