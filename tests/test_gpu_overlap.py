"""Kernels of one GPU that overlap the tail of the kernel in front (programmatic dependent launch), of different kinds in a
row: MoE dispatch and combine, the copy kernel of a single rank, plain GEMMs of each tile form.  The launches overlap, the
accesses must not: every chain gives the bytes of the same chain with a wait after every call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,hidden,inter,split,width", [(7, 512, 1024, 4, 32), (64, 2048, 4096, 0, 0), (700, 1024, 2048, 1, 224), (2500, 2048, 4096, 0, 512)])
@pytest.mark.parametrize("streams", [1, 2])
def test_mixed_chain_equals_the_chain_that_waits(tokens, hidden, inter, split, width, streams):
    import hcomm_b200 as hb
    from hcomm_b200 import _lib
    from hcomm_b200.ops.gemm import gemm_bf16, take_kernel_error
    from hcomm_b200.ops.moe import MoeExchange
    torch.cuda.set_device(0)
    lib = _lib.load()
    comm = hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=8)
    experts, topk = 16, 4
    moe = MoeExchange(comm, experts, topk, hidden, tokens, capacity_factor=1.0)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x0 = torch.randn(tokens, hidden, device="cuda", generator=g).to(torch.bfloat16)
    up = (torch.randn(inter, hidden, device="cuda", generator=g) / hidden ** 0.5).to(torch.bfloat16)
    down = (torch.randn(hidden, inter, device="cuda", generator=g) / inter ** 0.5).to(torch.bfloat16)
    idx = torch.rand(tokens, experts, device="cuda", generator=g).topk(topk, dim=1).indices.to(torch.int32).contiguous()
    gates = torch.rand(tokens, topk, device="cuda", generator=g)
    ballast = torch.randn(16 << 20, device="cuda", generator=g)         # 64 MB: the copy in front of a GEMM is longer than its set-up
    side = torch.cuda.Stream()

    def chain(wait):
        # buffers are written by one call and read by the next, and overwritten while their last reader has just been queued
        x, h = x0.clone(), torch.empty(tokens, inter, device="cuda", dtype=torch.bfloat16)
        y = torch.empty(tokens * topk, hidden, device="cuda", dtype=torch.bfloat16)
        out, copy = torch.empty_like(x), torch.empty_like(ballast)
        seen = []
        main, turn = torch.cuda.current_stream(), 0

        def call(fn):
            # two streams take turns, each call behind the event of the one in front
            nonlocal turn
            if streams == 2:
                here, before = (side, main) if turn % 2 == 0 else (main, side)
                here.wait_stream(before)
                turn += 1
                with torch.cuda.stream(here):
                    fn()
            else:
                fn()
            if wait:
                torch.cuda.synchronize()

        def experts_step(rec):
            n = tokens * topk
            y.copy_(rec.rows[:n])
            y.view(n, -1, 128).mul_(rec.scales[:n].to(torch.bfloat16).unsqueeze(-1))
        for _ in range(4):
            call(lambda: gemm_bf16(x, up, h))
            call(lambda: experts_step(moe.dispatch(x, idx)))            # dispatch behind a GEMM
            call(lambda: gemm_bf16(h, down, x))                         # overwrites what dispatch read
            call(lambda: moe.combine(y, gates, out))                    # combine behind a GEMM
            call(lambda: comm.all_reduce_scaled(out, x, 0.25))          # copy behind combine, over the GEMM's result
            call(lambda: moe.dispatch(x, idx))
            call(lambda: gemm_bf16(x, up, h))                           # GEMM behind a dispatch
            call(lambda: comm.all_reduce(ballast, copy))
            call(lambda: gemm_bf16(h, down, x))                         # GEMM behind a long copy
            if streams == 2 and turn % 2 == 1:
                call(lambda: None)
            seen.append((x.clone(), h.clone(), out.clone()))
        torch.cuda.synchronize()
        return seen
    lib.HcommGemmSetTuning(0, width)
    lib.HcommGemmSetSplit(split)
    try:
        want = chain(True)
        for _ in range(3):
            for a, b in zip(chain(False), want):
                assert all(torch.equal(u, v) for u, v in zip(a, b))
    finally:
        lib.HcommGemmSetTuning(0, 0)
        lib.HcommGemmSetSplit(0)
        moe.destroy()
    assert take_kernel_error() == 0 and comm.async_error() == 0
    comm.destroy()
