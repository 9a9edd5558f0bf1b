"""The rule that picks the plain GEMM's tile, on the CPU: every shape gets a tile that the kernels take."""
import ctypes

import pytest

from hcomm_b200 import _lib

CAPS = [(74, 33, 15), (74, 0, 0), (8, 4, 2), (1, 0, 0)]


def pick(m, n, k, caps):
    bn, split = ctypes.c_int(), ctypes.c_int()
    _lib.load().HcommToolGemmTile(m, n, k, *caps, ctypes.byref(bn), ctypes.byref(split))
    return bn.value, split.value


@pytest.mark.parametrize("caps", CAPS)
def test_every_shape_gets_a_tile_that_the_kernel_takes(caps):
    sizes = [8, 64, 72, 136, 256, 264, 1000, 1024, 3584, 4096, 5000, 8192, 28672, 128256]
    for m in [1, 2, 15, 31, 32, 33, 64, 65, 96, 127, 128, 200, 255, 256, 257, 300, 777, 1024, 5003, 8192, 100000]:
        for n in sizes:
            for k in sizes:
                bn, split = pick(m, n, k, caps)
                assert split in (1, 2, 4) and (split == 1 or caps[split // 2] > 0), (m, n, k, split)
                if bn == 512:
                    assert split == 1
                    continue
                assert 32 <= bn <= 256 and bn % 32 == 0, (m, n, k, bn)
                assert bn - 32 < m, "a tile with a whole step of empty columns"
                assert split == 1 or (k + 63) // 64 >= 4 * split, "a part of K that is hardly a step"


B200 = (74, 33, 22, 15)         # clusters of one to four pairs that one holds at once


def choice(m, n, k, caps=B200):
    """(kernel, tokens per tile, pairs that share a tile) on a device that holds so many clusters of one to four pairs."""
    bn, split = ctypes.c_int(), ctypes.c_int()
    kernel = _lib.load().HcommToolGemmTileOf(m, n, k, (ctypes.c_int * 4)(*caps), ctypes.byref(bn), ctypes.byref(split))
    return kernel, bn.value, split.value


@pytest.mark.parametrize("caps", [B200, (8, 4, 3, 2), (74, 0, 24, 0)])
def test_every_shape_gets_a_tile_where_three_pairs_may_share_one(caps):
    sizes = [8, 72, 136, 264, 768, 1000, 1024, 3584, 4096, 5000, 8192, 28672, 128256]
    shared = 0
    for m in [1, 15, 32, 33, 64, 65, 96, 127, 128, 129, 160, 200, 256, 257, 300, 777, 1024, 5003, 100000]:
        for n in sizes:
            for k in sizes:
                kernel, bn, split = choice(m, n, k, caps)
                assert 1 <= split <= 4 and (split == 1 or caps[split - 1] > 0), (m, n, k, split)
                if kernel != 0:
                    assert split == 1 and bn == {1: 512, 2: 128, 3: 224}[kernel]
                    continue
                assert 32 <= bn <= 256 and bn % 32 == 0 and bn - 32 < m, (m, n, k, bn)
                if split > 1:
                    assert (k + 63) // 64 >= 4 * split, "a part of K that is hardly a step"
                    assert -(-n // 256) * -(-m // bn) <= caps[split - 1], "shared tiles in more than one wave"
                    assert split != 3 or m <= 128, "three pairs beyond what they were measured to win"
                    shared += split == 3
    assert shared > 0


def test_known_choices_of_a_b200():
    # as on devices without clusters of three pairs, below, but for the shapes that three pairs win
    for m, n, k, kernel, bn, split in [(16, 8192, 28672, 0, 32, 2), (16, 28672, 8192, 0, 32, 1), (96, 3584, 8192, 0, 96, 4), (33, 128256, 4096, 0, 64, 1),
                                       (8192, 28672, 8192, 1, 512, 1), (777, 14336, 4096, 0, 160, 1), (8192, 3584, 8192, 0, 224, 1), (65536, 4096, 64, 1, 512, 1),
                                       (16384, 8, 256, 2, 128, 1), (5956, 24, 936, 2, 128, 1), (512, 14336, 8192, 3, 224, 1)]:
        assert choice(m, n, k) == (kernel, bn, split), (m, n, k)
    # us with three pairs, and with what is taken without: 10.0 and 10.1, 10.4 and 11.4, 24.2 and 25.9
    for m, n, k, bn, without in [(40, 4096, 4096, 64, (64, 2)), (64, 4096, 4096, 64, (32, 2)), (96, 4096, 14336, 96, (96, 2))]:
        assert choice(m, n, k) == (0, bn, 3), (m, n, k)
        assert choice(m, n, k, (74, 33, 0, 15)) == (0, *without), (m, n, k)
    # limits of three pairs: tokens, steps of K, one wave
    assert choice(128, 4096, 14336)[2] == 3 and choice(129, 4096, 14336)[2] != 3
    assert choice(16, 4096, 14336, (74, 33, 15, 15))[2] != 3 and choice(16, 5000, 11 * 64)[2] != 3


def test_known_choices():
    caps = (74, 33, 15)
    assert pick(16, 8192, 28672, caps) == (32, 2)       # 32 tiles: two pairs each, so that enough SMs ask for the weights
    assert pick(16, 28672, 8192, caps) == (32, 1)       # 112 tiles keep the chip busy as they are
    assert pick(96, 3584, 8192, caps) == (96, 4)        # 14 tiles, a deep K
    assert pick(33, 128256, 4096, caps) == (64, 1)      # one tile across all tokens: every weight is fetched once
    assert pick(40, 4096, 4096, caps) == (64, 2)        # not two token tiles that both read every weight
    assert pick(8192, 28672, 8192, caps) == (512, 1)    # 25 full waves: the least operand traffic
    assert pick(777, 14336, 4096, caps) == (160, 1)     # 800 columns of work for 777 tokens
    assert pick(8192, 3584, 8192, caps) == (224, 1)     # seven full waves instead of eight of 256 columns


def test_shallow_k_takes_wide_tiles():
    caps = (74, 33, 15)
    # emptying the accumulators bounds these: measured 119 us (310 with 64 tokens), 7.6 (21 with 32), 11.8 (36 with 32), 10.1 (15.5)
    assert pick(65536, 4096, 64, caps) == (512, 1)
    assert pick(8192, 1024, 64, caps) == (512, 1)
    assert pick(1000, 14336, 64, caps) == (512, 1)
    assert pick(16384, 512, 136, caps)[0] >= 160
    # operands whose rows straddle lines, many waves: 107 us (122 with 256)
    assert pick(16384, 4096, 1000, caps) == (512, 1)
    # 48 clusters of four would come in two waves: 95.7 us with 128/1, 112 with 192/2
    assert pick(1101, 4096, 14336, caps)[1] == 1


def test_few_columns_of_many_rows_run_without_pairs():
    caps = (74, 33, 15)
    kernel = _lib.load().HcommToolGemmKernel
    assert kernel(16384, 8, 256, *caps) == 2 and kernel(8192, 64, 512, *caps) == 2 and kernel(65536, 8, 64, *caps) == 2
    assert kernel(5956, 24, 936, *caps) == 2
    # too few rows, too deep a K, too many columns
    assert kernel(1000, 8, 256, *caps) == 0 and kernel(16384, 8, 4096, *caps) == 0 and kernel(65536, 8, 1000, *caps) == 0
    assert kernel(16384, 136, 256, *caps) != 2 and kernel(8192, 28672, 8192, *caps) == 1


def test_round_batches_of_layers_224_wide():
    caps = (74, 33, 15)
    kernel = _lib.load().HcommToolGemmKernel
    assert kernel(512, 14336, 8192, *caps) == 3 and kernel(2048, 14336, 8192, *caps) == 3 and kernel(512, 7168, 8192, *caps) == 3
    # not a multiple of 256 tokens or of 224 weights, a shallower K, whole waves anyway
    assert kernel(511, 14336, 8192, *caps) != 3 and kernel(512, 8192, 8192, *caps) != 3 and kernel(4096, 14336, 1024, *caps) != 3
    assert kernel(8192, 28672, 8192, *caps) == 1


@pytest.mark.parametrize("group", [0, 1, 3, 1000, 1 << 28, 1 << 30, 2147483647])
@pytest.mark.parametrize("m,n,width", [(1000, 5000, 256), (33, 128256, 64), (700, 256, 32), (8192, 8, 224)])
def test_every_tile_is_walked_once_whatever_group_is_asked_for(m, n, width, group):
    lib = _lib.load()
    wb, tb = ctypes.c_int(), ctypes.c_int()
    lib.HcommGemmSetTuning(group, 0)
    try:
        total = lib.HcommToolGemmOrder(m, n, 4096, width, -1, None, None)
        blocks_w, blocks_t = -(-n // 256), -(-m // width)
        assert total == blocks_w * blocks_t
        seen = set()
        for t in range(total):
            lib.HcommToolGemmOrder(m, n, 4096, width, t, ctypes.byref(wb), ctypes.byref(tb))
            assert 0 <= wb.value < blocks_w and 0 <= tb.value < blocks_t
            seen.add((wb.value, tb.value))
        assert len(seen) == total
    finally:
        lib.HcommGemmSetTuning(0, 0)
