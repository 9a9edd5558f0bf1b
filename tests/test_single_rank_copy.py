"""The copy kernel of a single rank: words of 16 bytes whatever element the buffers start on, the ends element by element."""
import ctypes

import pytest


@pytest.mark.parametrize("bytes_", list(range(0, 140)) + [3071, 3072, 3073, 49152 + 5, 1 << 20])
def test_split_reads_and_writes_inside_the_operand(bytes_):
    from hcomm_b200 import _lib
    lib = _lib.load()
    head, words, delta = ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_uint32()
    for i in range(16):
        for o in range(16):
            src, dst = 4096 + i, 8192 + o
            lib.HcommToolLocalSplit(ctypes.c_uint64(src), ctypes.c_uint64(dst), ctypes.c_uint64(bytes_), ctypes.byref(head), ctypes.byref(words), ctypes.byref(delta))
            h, w, d = head.value, words.value, delta.value
            tail = bytes_ - h - 16 * w
            assert 0 <= tail
            if w == 0:
                assert h == 0 and d == 0 and tail < 64
                continue
            assert h < 32 and tail < 32 and d < 16
            first = src + h - d                     # the words of the source: one more than of the result where they are shifted
            assert (dst + h) % 16 == 0 and first % 16 == 0
            assert first >= src and first + 16 * (w + (d > 0)) <= src + bytes_


def test_ctas():
    from hcomm_b200 import _lib
    ctas = _lib.load().HcommToolLocalCtas

    def of(bytes_, shifted=0, sms=148):
        return ctas(ctypes.c_uint64(bytes_), shifted, sms)
    assert [of(b) for b in (0, 1, 8192, 8193, 1 << 18)] == [1, 1, 1, 2, 32]
    # as many as leave SMs to the next call, while they hold the operand in one round
    assert of(1 << 20) == of(2 << 20) == of(3 << 20) == of(1 << 20, 1) == 64 and of(1 << 20, 0, 20) == 20
    assert of((3 << 20) + 1) == of((160 << 20) - 1) == of((3 << 20) + 1, 1) == 148
    # more rounds for the largest ones whose buffers start alike
    assert of(160 << 20) == of(1 << 40) == 592 and of(1 << 28, 1) == 148


@pytest.mark.gpu
@pytest.mark.parametrize("name,size", [("uint8", 1), ("bfloat16", 2), ("float32", 4), ("float64", 8)])
def test_every_shift_between_the_buffers(name, size):
    import torch

    import hcomm_b200 as hb
    dtype = getattr(torch, name)
    torch.cuda.set_device(0)
    comm = hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=4)
    try:
        g = torch.Generator(device="cuda").manual_seed(size)
        steps = 16 // size
        # what a warp takes at a time: six words of each lane, and eight of the shifted ones but 16-bit types; 16 warps of a CTA per SM
        pieces = {3072 // size, 4096 // size}
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        # no whole word; a piece and its neighbours; the last size that few CTAs take, and the first that all do; two and three rounds
        # of all of them and an odd rest, in either kernel's pieces
        counts = {1, 3 * steps, (3 << 20) // size, (3 << 20) // size + 1}
        for piece in pieces:
            counts |= {piece - 1, piece, piece + steps + 1}
        for words in (6, 8):
            counts |= {rounds * sms * 16 * words * 512 // size + 3 * 4096 // size + 5 for rounds in (1, 2)}
        for count in sorted(counts):
            base = torch.randint(-100, 100, (count + 32,), device="cuda", generator=g).to(dtype)
            for i in range(0, steps, max(1, steps // 8)):
                for o in (0, 1, steps - 1):
                    x = base[i:i + count]
                    out = torch.full((count + 32,), 7, device="cuda", dtype=dtype)
                    want = out.clone()
                    want[o:o + count] = x
                    comm.all_gather(x, out[o:o + count])
                    assert torch.equal(out, want), (count, i, o)
                    if dtype.is_floating_point:
                        comm.all_reduce_scaled(x, out[o:o + count], 0.5)       # exact
                        want[o:o + count] = x * 0.5
                        assert torch.equal(out, want), (count, i, o)
    finally:
        comm.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("name,size", [("uint8", 1), ("bfloat16", 2), ("float32", 4)])
def test_the_largest_operands_take_more_ctas(name, size):
    import torch

    import hcomm_b200 as hb
    dtype = getattr(torch, name)
    torch.cuda.set_device(0)
    comm = hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=4)
    try:
        g = torch.Generator(device="cuda").manual_seed(size)
        for count in ((160 << 20) // size - 1, (160 << 20) // size, (201 << 20) // size + 7):
            base = torch.randint(-100, 100, (count + 32,), device="cuda", generator=g).to(dtype)
            for i, o in ((0, 0), (5, 5), (0, 3)):           # alike, alike off a word, differently
                x = base[i:i + count]
                out = torch.full((count + 32,), 7, device="cuda", dtype=dtype)
                comm.all_gather(x, out[o:o + count])
                assert torch.equal(out[o:o + count], x) and bool((out[:o] == 7).all()) and bool((out[o + count:] == 7).all()), (count, i, o)
                if dtype.is_floating_point:
                    comm.all_reduce_scaled(x, out[o:o + count], 0.5)           # exact
                    assert torch.equal(out[o:o + count], x * 0.5) and bool((out[o + count:] == 7).all()), (count, i, o)
    finally:
        comm.destroy()
