"""Numerics of the tcgen05 GEMM against a plain PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 256, 512), (256, 512, 256), (1024, 1024, 1024), (384, 128, 192), (200, 136, 72),
                                   (2048, 3584, 1024)])
def test_gemm_matches_fp32_reference(m, n, k):
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    torch.manual_seed(m * 7 + n * 3 + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(n, k, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    c = gemm_bf16(a, b)
    torch.cuda.synchronize()
    assert take_kernel_error() == 0
    ref = a.float() @ b.float().t()
    err = (c.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * max(scale, 1.0), f"max abs err {err} vs scale {scale}"


def test_gemm_strided_operands():
    from hcomm_b200.ops.gemm import gemm_bf16
    a_full = torch.randn(256, 1024, device="cuda", dtype=torch.bfloat16)
    b_full = torch.randn(512, 1024, device="cuda", dtype=torch.bfloat16)
    a, b = a_full[:, 256:768], b_full[:, 256:768]   # K slice: pitch 1024, 512 columns used
    c = gemm_bf16(a, b)
    ref = a.float() @ b.float().t()
    assert torch.allclose(c.float(), ref, atol=0.5, rtol=2e-2)


@pytest.mark.parametrize("m,n,k,group", [(512, 1024, 256, 0), (2048, 4096, 1032, 0), (4096, 8192, 512, 12), (256, 512, 72, 1)])
def test_wide_tile_kernel_matches_fp32_reference(m, n, k, group):
    # 256 x 512 tiles (one accumulator, TMA-store epilogue) forced for shapes the selection rule would give narrower tiles,
    # including more tiles than CTA pairs, a K that is not a multiple of the 64-wide block, and a strided result
    from hcomm_b200 import _lib
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    lib = _lib.load()
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = (torch.randn(n, k, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    out_full = torch.zeros(m, n + 64, device="cuda", dtype=torch.bfloat16)
    out = out_full[:, :n]                       # pitch n + 64: the columns beyond n must stay untouched
    lib.HcommGemmSetTuning(group, 512)
    try:
        gemm_bf16(a, b, out)
        torch.cuda.synchronize()
    finally:
        lib.HcommGemmSetTuning(0, 0)
    assert take_kernel_error() == 0
    ref = a.float() @ b.float().t()
    err = (out.float() - ref).abs().max().item()
    assert err <= 1e-2 * max(ref.abs().max().item(), 1.0), f"max abs err {err}"
    assert out_full[:, n:].abs().max().item() == 0


@pytest.mark.parametrize("width,split", [(32, 1), (32, 4), (96, 1), (96, 2), (224, 1), (224, 4), (256, 1), (256, 2), (256, 4), (512, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 136, 264), (33, 264, 512), (200, 1000, 520), (257, 776, 1032), (700, 2048, 320)])
def test_gemm_tiles_and_parts_of_k(m, n, k, width, split):
    # rows and columns around the edges of the tiles, K not a multiple of the 64-wide step or of the parts of a split,
    # a result inside a wider matrix whose other columns must stay as they are, and bit-equal results from run to run
    from hcomm_b200 import _lib
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    lib = _lib.load()
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    b = (torch.randn(n, k, device="cuda") * 0.05).to(torch.bfloat16)
    full = torch.full((2, m, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    lib.HcommGemmSetTuning(0, width)
    lib.HcommGemmSetSplit(split)
    try:
        for i in range(2):
            gemm_bf16(a, b, full[i][:, :n])
        torch.cuda.synchronize()
    finally:
        lib.HcommGemmSetTuning(0, 0)
        lib.HcommGemmSetSplit(0)
    assert take_kernel_error() == 0
    assert torch.equal(full[0], full[1]) and bool((full[:, :, n:] == 7.0).all())
    ref = a.double() @ b.double().t()
    # one rounding to bf16 (half a step, 2^-9) and fp32 sums of k products (k * 2^-24 of the sum of magnitudes)
    bound = 2.0 ** -8 * ref.abs() + k * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t())
    assert bool(((full[0][:, :n].double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("m,h,i", [(16, 1024, 4096), (300, 1024, 2048), (2048, 8192, 8192)])
def test_back_to_back_calls_see_each_others_results(m, h, i):
    # a chain in which every call reads what the call in front wrote and overwrites what it read: the launches overlap,
    # the accesses must not
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    torch.manual_seed(m)
    up = (torch.randn(i, h, device="cuda") / h ** 0.5).to(torch.bfloat16)
    down = (torch.randn(h, i, device="cuda") / i ** 0.5).to(torch.bfloat16)
    x0 = torch.randn(m, h, device="cuda").to(torch.bfloat16)

    def chain(wait):
        x, y = x0.clone(), torch.empty(m, i, device="cuda", dtype=torch.bfloat16)
        for _ in range(6):
            gemm_bf16(x, up, y)
            if wait:
                torch.cuda.synchronize()
            gemm_bf16(y, down, x)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return x
    want = chain(True)
    for _ in range(3):
        assert torch.equal(chain(False), want)
    assert take_kernel_error() == 0


@pytest.mark.parametrize("width", [32, 256, 512])
def test_oversized_raster_group(width):
    from hcomm_b200 import _lib
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    lib = _lib.load()
    a = torch.randn(1000, 256, device="cuda").to(torch.bfloat16)
    b = torch.randn(776, 256, device="cuda").to(torch.bfloat16)
    lib.HcommGemmSetTuning(0, width)
    want = gemm_bf16(a, b)
    try:
        lib.HcommGemmSetTuning(1 << 30, width)          # times the number of token blocks this is no 32-bit number
        got = gemm_bf16(a, b)
        torch.cuda.synchronize()
    finally:
        lib.HcommGemmSetTuning(0, 0)
    assert take_kernel_error() == 0 and torch.equal(got, want)


def device_caps():
    """Clusters of one to four CTA pairs that the current device holds at once: what its choices go by."""
    import ctypes

    from hcomm_b200 import _lib
    caps = (ctypes.c_int * 4)()
    _lib.load().HcommToolGemmCaps(caps)
    return caps


def test_the_device_holds_clusters_of_every_number_of_pairs():
    caps = list(device_caps())
    # a pair fills two SMs
    assert all(n > 0 for n in caps) and all(caps[i] * (i + 1) <= caps[0] for i in range(4)) and caps[0] >= caps[1] >= caps[2] >= caps[3]


@pytest.mark.parametrize("m,n,k", [(4097, 8, 64), (12800, 128, 8), (5003, 72, 136), (8192, 24, 1000), (19000, 8, 72), (40001, 64, 512)])
def test_few_columns_of_many_rows(m, n, k):
    # the kernel without pairs is the one that runs here; rows of a longer pitch in, a result inside a wider matrix
    from hcomm_b200 import _lib
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    assert _lib.load().HcommToolGemmTileOf(m, n, k, device_caps(), None, None) == 2
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :k]
    b = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    full = torch.full((m, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm_bf16(a, b, full[:, :n])
    torch.cuda.synchronize()
    assert take_kernel_error() == 0 and bool((full[:, n:] == 7.0).all())
    ref = a.double() @ b.double().t()
    # one rounding to bf16 (half a step, 2^-9) and fp32 sums of k products (k * 2^-24 of the sum of magnitudes)
    bound = 2.0 ** -8 * ref.abs() + k * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t())
    assert bool(((full[:, :n].double() - ref).abs() <= bound).all())


def test_round_batch_of_a_layer_224_wide():
    # 256 x 224 tiles with the tokens as rows, operands and result of a longer pitch
    from hcomm_b200 import _lib
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    m, n, k = 512, 14336, 4104
    assert _lib.load().HcommToolGemmTileOf(m, n, k, device_caps(), None, None) == 3
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :k]
    b = (torch.randn(n, k + 16, device="cuda", generator=g) * 0.05).to(torch.bfloat16)[:, :k]
    full = torch.full((m, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    for _ in range(2):          # the second call behind the first
        gemm_bf16(a, b, full[:, :n])
    torch.cuda.synchronize()
    assert take_kernel_error() == 0 and bool((full[:, n:] == 7.0).all())
    ref = a.double() @ b.double().t()
    # one rounding to bf16 (half a step, 2^-9) and fp32 sums of k products (k * 2^-24 of the sum of magnitudes)
    bound = 2.0 ** -8 * ref.abs() + k * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t())
    assert bool(((full[:, :n].double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("m,n,k", [(1, 4096, 1000), (33, 1032, 4096), (128, 3584, 1000), (160, 4096, 1024), (129, 776, 2056), (257, 264, 520)])
@pytest.mark.parametrize("split", [1, 2, 3, 4])
def test_every_number_of_parts_of_k(m, n, k, split):
    from hcomm_b200 import _lib
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a = torch.randn(m, k + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :k]
    b = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    full = torch.full((m, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    lib = _lib.load()
    assert device_caps()[split - 1] > 0             # or the forced number would be left out
    ref = a.double() @ b.double().t()
    # one rounding to bf16 (half a step, 2^-9) and fp32 sums of k products (k * 2^-24 of the sum of magnitudes)
    bound = 2.0 ** -8 * ref.abs() + k * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t())
    try:
        for width in (32, 96, 160, 192):
            lib.HcommGemmSetTuning(0, width)
            lib.HcommGemmSetSplit(split)
            for _ in range(2):          # the second call behind the first
                full.fill_(7.0)
                gemm_bf16(a, b, full[:, :n])
                gemm_bf16(a, b, full[:, :n])
            torch.cuda.synchronize()
            assert take_kernel_error() == 0 and bool((full[:, n:] == 7.0).all())
            assert bool(((full[:, :n].double() - ref).abs() <= bound).all()), width
    finally:
        lib.HcommGemmSetTuning(0, 0)
        lib.HcommGemmSetSplit(0)
