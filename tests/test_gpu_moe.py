"""MoE dispatch / combine kernels, ranks sharing one GPU, against a PyTorch reference of the same routing."""
import pytest
import torch

from helpers import run_ranks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,experts,topk,hidden,tokens", [(2, 8, 2, 512, 64), (4, 16, 4, 1024, 96), (2, 32, 8, 7168, 128)])
def test_dispatch_and_combine(n, experts, topk, hidden, tokens):
    import hcomm_b200 as hb
    from hcomm_b200.ops.moe import MoeExchange, quantize_e4m3_1x128
    info = hb.get_root_info()

    def init(r):
        torch.cuda.set_device(0)
        return hb.Communicator(n, info, r, buffer_mb=8)
    comms = run_ranks(n, init)
    moes = run_ranks(n, lambda r: (torch.cuda.set_device(0), MoeExchange(comms[r], experts, topk, hidden, tokens))[1])
    try:
        epr = experts // n
        g = torch.Generator(device="cuda").manual_seed(7)
        xs = [torch.randn(tokens, hidden, device="cuda", generator=g).to(torch.bfloat16) for _ in range(n)]
        idx = [torch.stack([torch.randperm(experts, device="cuda", generator=g)[:topk] for _ in range(tokens)]).to(torch.int32).contiguous() for _ in range(n)]
        gates = [torch.rand(tokens, topk, device="cuda", generator=g).float().contiguous() for _ in range(n)]
        outs = [None] * n
        recv_snap = [None] * n
        for rep in range(2):
            def op(r):
                torch.cuda.set_device(0)
                rec = moes[r].dispatch(xs[r], idx[r])
                torch.cuda.synchronize()
                nrows = rec.num_rows
                recv_snap[r] = (rec.rows[:nrows].clone(), rec.scales[:nrows].clone(), rec.origin[:nrows].clone(), rec.expert_offsets.clone())
                # "expert": y = 2 * dequantised row + local expert index
                deq = rec.dequantized(nrows)
                offs = rec.expert_offsets.tolist()
                y = torch.empty(nrows, hidden, device="cuda", dtype=torch.bfloat16)
                for el in range(epr):
                    y[offs[el]:offs[el + 1]] = (2 * deq[offs[el]:offs[el + 1]] + el).to(torch.bfloat16)
                outs[r] = moes[r].combine(y, gates[r])
                torch.cuda.synchronize()
            run_ranks(n, op)
            assert all(m.overflow() == 0 for m in moes)
            for r in range(n):
                rows, scales, origin, offs = recv_snap[r]
                offs = offs.tolist()
                expected_total = sum(int(((idx[s] // epr) == r).sum().item()) for s in range(n))
                assert offs[-1] == expected_total
                for el in range(epr):
                    e = r * epr + el
                    seg = slice(offs[el], offs[el + 1])
                    src_rank = (origin[seg] >> 32).tolist()
                    tk = (origin[seg] & 0xffffffff).tolist()
                    assert src_rank == sorted(src_rank), "rows of one expert are grouped by source rank"
                    want = sorted((s, int(t) * topk + int(k)) for s in range(n) for t, k in (idx[s] == e).nonzero().tolist())
                    assert sorted(zip(src_rank, tk)) == want
                    for i, (s, key) in enumerate(zip(src_rank, tk)):
                        if i % 7:      # spot-check rows
                            continue
                        q, sc = quantize_e4m3_1x128(xs[s][key // topk:key // topk + 1])
                        assert torch.equal(rows[offs[el] + i].view(torch.uint8), q[0].view(torch.uint8))
                        assert torch.allclose(scales[offs[el] + i], sc[0])
            for r in range(n):
                q, sc = quantize_e4m3_1x128(xs[r])
                deq = (q.float().view(tokens, -1, 128) * sc.unsqueeze(-1)).view(tokens, hidden)
                ref = torch.zeros(tokens, hidden, device="cuda")
                for k in range(topk):
                    el = (idx[r][:, k] % epr).float().unsqueeze(1)
                    ref += gates[r][:, k:k + 1] * (2 * deq + el).to(torch.bfloat16).float()
                err = (outs[r].float() - ref).abs().max().item()
                assert err <= 3e-2 * max(1.0, ref.abs().max().item()), (rep, r, err)
    finally:
        run_ranks(n, lambda r: moes[r].destroy())
        run_ranks(n, lambda r: comms[r].destroy())


@pytest.mark.parametrize("capacity_factor,masked", [(2.0, True), (0.3, False)])
def test_masked_experts_and_dropped_rows_stay_out_of_the_sum(capacity_factor, masked):
    """An expert index outside the range masks that choice, and rows beyond the receive capacity are dropped: combine must
    add neither - the landing slot of such a (token, k) holds whatever an earlier step left there."""
    import hcomm_b200 as hb
    from hcomm_b200.ops.moe import MoeExchange, quantize_e4m3_1x128
    n, experts, topk, hidden, tokens = 2, 8, 4, 512, 64
    info = hb.get_root_info()

    def init(r):
        torch.cuda.set_device(0)
        return hb.Communicator(n, info, r, buffer_mb=8)
    comms = run_ranks(n, init)
    moes = run_ranks(n, lambda r: (torch.cuda.set_device(0), MoeExchange(comms[r], experts, topk, hidden, tokens, capacity_factor=capacity_factor))[1])
    try:
        g = torch.Generator(device="cuda").manual_seed(3)
        xs = [torch.randn(tokens, hidden, device="cuda", generator=g).to(torch.bfloat16) for _ in range(n)]
        gates = [torch.rand(tokens, topk, device="cuda", generator=g).float().contiguous() for _ in range(n)]
        outs, sent = [None] * n, [None] * n
        for step in range(2):
            # step 0 fills every landing slot with large values (nothing masked), step 1 is the one that is checked
            idx = [torch.stack([torch.randperm(experts, device="cuda", generator=g)[:topk] for _ in range(tokens)]).to(torch.int32).contiguous() for _ in range(n)]
            if masked and step == 1:
                for r in range(n):
                    idx[r][::3, 1] = -1
                    idx[r][1::5, 3] = experts + 7
            scale = 1000.0 if step == 0 else 1.0

            def op(r):
                torch.cuda.set_device(0)
                rec = moes[r].dispatch(xs[r], idx[r])
                torch.cuda.synchronize()
                nrows = rec.num_rows
                offs = rec.expert_offsets.tolist()
                assert all(0 <= o <= moes[r].layout.maxRecvRows for o in offs) and offs == sorted(offs)
                y = (rec.dequantized(nrows) * scale).to(torch.bfloat16)
                outs[r] = moes[r].combine(y, gates[r])
                torch.cuda.synchronize()
                sent[r] = moes[r].sent[:tokens].clone()
            run_ranks(n, op)
            dropped = sum(m.overflow() for m in moes)
            if step == 0:
                continue
            if capacity_factor < 1:
                assert dropped > 0, "the capacity was meant to overflow"
            for r in range(n):
                in_range = (idx[r] >= 0) & (idx[r] < experts)
                assert torch.all(sent[r].bool() <= in_range), "a masked choice was marked as sent"
                if capacity_factor >= 1:
                    assert torch.equal(sent[r].bool(), in_range)
                q, sc = quantize_e4m3_1x128(xs[r])
                deq = (q.float().view(tokens, -1, 128) * sc.unsqueeze(-1)).view(tokens, hidden).to(torch.bfloat16).float()
                ref = deq * (gates[r] * sent[r].float()).sum(dim=1, keepdim=True)
                assert torch.isfinite(outs[r].float()).all()
                err = (outs[r].float() - ref).abs().max().item()
                assert err <= 3e-2 * max(1.0, ref.abs().max().item()), (r, err)
    finally:
        run_ranks(n, lambda r: moes[r].destroy())
        run_ranks(n, lambda r: comms[r].destroy())


@pytest.mark.parametrize("experts,topk,hidden,tokens,capacity_factor,masked", [
    (8, 2, 512, 1, 1.0, False), (8, 16, 512, 33, 1.0, False), (256, 8, 7168, 64, 1.0, True), (1024, 4, 8192, 300, 1.0, True), (64, 6, 2048, 1999, 1.0, False),
    (16, 4, 1024, 700, 0.4, True)])
def test_single_rank_rows_are_summed_where_the_experts_wrote_them(experts, topk, hidden, tokens, capacity_factor, masked):
    """One rank: every row stays local.  Dispatched bytes, offsets and marks against the reference quantiser, the sum bit for
    bit against fp32 accumulation in the order of k; CTAs with no token, several claim rounds per CTA, one to many segments."""
    import hcomm_b200 as hb
    from hcomm_b200.ops.moe import MoeExchange, quantize_e4m3_1x128
    torch.cuda.set_device(0)
    comm = hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=8)
    moe = MoeExchange(comm, experts, topk, hidden, tokens, capacity_factor=capacity_factor)
    try:
        g = torch.Generator(device="cuda").manual_seed(tokens)
        for t in (tokens, max(1, tokens // 3)):         # fewer tokens than the exchange is made for, over older contents
            x = torch.randn(t, hidden, device="cuda", generator=g).to(torch.bfloat16)
            # with replacement: several choices of one token may name the same expert
            idx = torch.randint(0, experts, (t, topk), device="cuda", generator=g).to(torch.int32)
            if masked:
                idx[torch.rand(t, topk, device="cuda", generator=g) < 0.2] = -1
                idx[0, 0] = experts
            gates = torch.rand(t, topk, device="cuda", generator=g)
            rec = moe.dispatch(x, idx)
            torch.cuda.synchronize()
            inside = (idx >= 0) & (idx < experts)
            counts = torch.bincount(idx[inside].long(), minlength=experts)
            want = torch.cat([torch.zeros(1, device="cuda", dtype=torch.int64), counts.cumsum(0)]).clamp(max=moe.layout.maxRecvRows)
            assert torch.equal(rec.expert_offsets.long(), want)
            sent, n = moe.sent[:t].bool(), rec.num_rows
            assert bool((sent <= inside).all()) and int(sent.sum()) == n and moe.overflow() == int(inside.sum()) - n
            origin = rec.origin[:n]
            assert torch.equal(origin.sort().values, sent.flatten().nonzero().flatten())
            expert_of_row = torch.bucketize(torch.arange(n, device="cuda"), want[1:], right=True)
            assert torch.equal(idx.flatten()[origin].long(), expert_of_row)
            q, sc = quantize_e4m3_1x128(x)
            assert torch.equal(rec.rows[:n].view(torch.uint8), q.view(torch.uint8)[origin // topk]) and torch.equal(rec.scales[:n], sc[origin // topk])
            y = torch.randn(n, hidden, device="cuda", generator=g).to(torch.bfloat16)
            out = moe.combine(y, gates)
            row = torch.full((t * topk,), -1, device="cuda", dtype=torch.int64)
            row[origin] = torch.arange(n, device="cuda")
            acc = torch.zeros(t, hidden, device="cuda", dtype=torch.float64)
            for k in range(topk):                       # a fused multiply-add rounds once: the product is exact in fp64, the sum is rounded to fp32
                r = row.view(t, topk)[:, k]
                step = (acc + gates[:, k:k + 1].double() * y[r.clamp(min=0)].double()).float().double()
                acc = torch.where((r >= 0).unsqueeze(1), step, acc)
            assert torch.equal(out, acc.float().to(torch.bfloat16))
    finally:
        moe.destroy()
        comm.destroy()


def test_combine_of_more_tokens_than_were_dispatched_adds_nothing_for_the_rest():
    """The marks and rows of tokens beyond the last dispatch are an older one's, and the experts' output holds none of those
    rows: their sums are zero, whatever the older dispatch left behind."""
    import hcomm_b200 as hb
    from hcomm_b200.ops.moe import MoeExchange
    torch.cuda.set_device(0)
    comm = hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=8)
    moe = MoeExchange(comm, 8, 2, 512, 64)
    try:
        x = torch.randn(64, 512, device="cuda").to(torch.bfloat16)
        idx = torch.randint(0, 8, (64, 2), device="cuda").to(torch.int32)
        moe.dispatch(x, idx)
        moe.dispatch(x[:5].contiguous(), idx[:5].contiguous())
        out = moe.combine(torch.ones(10, 512, device="cuda", dtype=torch.bfloat16), torch.ones(64, 2, device="cuda"))
        torch.cuda.synchronize()
        assert bool((out[:5] == 2).all()) and bool((out[5:] == 0).all())
    finally:
        moe.destroy()
        comm.destroy()


@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("hidden,tokens", [(512, 5), (1024, 300)])
def test_result_inside_the_experts_output_and_rows_in_the_landing_area(n, hidden, tokens):
    """A result that overlaps the experts' output overwrites rows that other tokens still need: the sum is the one that a
    result elsewhere gets, wherever in y it lies.  And a caller that asks for the landing area finds every row that was sent
    in its slot (token, k), those of its own rank's experts too."""
    import ctypes
    import hcomm_b200 as hb
    from hcomm_b200 import _lib
    from hcomm_b200.ops.moe import MoeExchange, _view
    experts, topk = 8, 4
    info = hb.get_root_info()

    def init(r):
        torch.cuda.set_device(0)
        return hb.Communicator(n, info, r, buffer_mb=8)
    comms = run_ranks(n, init)
    moes = run_ranks(n, lambda r: (torch.cuda.set_device(0), MoeExchange(comms[r], experts, topk, hidden, tokens, capacity_factor=2.0))[1])
    try:
        g = torch.Generator(device="cuda").manual_seed(hidden)
        xs = [torch.randn(tokens, hidden, device="cuda", generator=g).to(torch.bfloat16) for _ in range(n)]
        idx = [torch.rand(tokens, experts, device="cuda", generator=g).topk(topk, dim=1).indices.to(torch.int32).contiguous() for _ in range(n)]
        gates = [torch.rand(tokens, topk, device="cuda", generator=g) for _ in range(n)]
        idx[0][::3, 1] = -1
        want, slots = [None] * n, [None] * n

        def plain(r):
            torch.cuda.set_device(0)
            rec = moes[r].dispatch(xs[r], idx[r])
            torch.cuda.synchronize()
            y = rec.dequantized().to(torch.bfloat16)
            want[r] = moes[r].combine(y, gates[r])
            torch.cuda.synchronize()
        run_ranks(n, plain)

        for where in ("start", "middle", "end"):
            def inside(r):
                torch.cuda.set_device(0)
                rec = moes[r].dispatch(xs[r], idx[r])
                torch.cuda.synchronize()
                rows = rec.num_rows
                y = torch.zeros(max(rows, tokens) + tokens, hidden, device="cuda", dtype=torch.bfloat16)
                y[:rows] = rec.dequantized(rows).to(torch.bfloat16)
                at = {"start": 0, "middle": rows // 3, "end": max(0, rows - tokens)}[where]
                out = moes[r].combine(y, gates[r], out=y[at:at + tokens])
                torch.cuda.synchronize()
                assert torch.equal(out, want[r]), where
            run_ranks(n, inside)

        def asked(r):
            torch.cuda.set_device(0)
            ptr = ctypes.c_void_p()
            assert _lib.load().HcommMoeGetBuffers(moes[r]._h, None, None, None, None, ctypes.byref(ptr)) == 0
            rec = moes[r].dispatch(xs[r], idx[r])
            torch.cuda.synchronize()
            out = moes[r].combine(rec.dequantized().to(torch.bfloat16), gates[r])
            torch.cuda.synchronize()
            assert torch.equal(out, want[r])
            slots[r] = _view(ptr.value, (tokens, topk, hidden), torch.bfloat16, torch.device("cuda", 0)).clone()
        run_ranks(n, asked)
        for r in range(n):
            q = moes[r].sent[:tokens].bool()
            # every expert here returns the dequantised token, so each slot that was sent holds it
            from hcomm_b200.ops.moe import quantize_e4m3_1x128
            f8, sc = quantize_e4m3_1x128(xs[r])
            row = (f8.float().view(tokens, -1, 128) * sc.unsqueeze(-1)).view(tokens, 1, hidden).to(torch.bfloat16)
            assert bool(q.any()) and torch.equal(slots[r][q], row.expand(-1, topk, -1)[q])
    finally:
        run_ranks(n, lambda r: moes[r].destroy())
        run_ranks(n, lambda r: comms[r].destroy())


@pytest.mark.parametrize("experts,topk,hidden,tokens,masked", [
    (256, 8, 7168, 1, False),           # a token, one CTA
    (8, 1, 512, 17000, True),           # as many choices as every CTA counts alone, and one more
    (8, 1, 512, 17001, True),
    (64, 3, 2048, 8001, True),          # in pairs, whose threads do not come out even in choices of a token
    (8, 1, 8192, 6714, False),          # in pairs for what there is to move
    (256, 8, 7168, 4145, True),         # the pairs' tokens do not come out even
    (1024, 16, 512, 9600, False),       # a CTA claims rows twice, all counters
    (1024, 16, 512, 560, True),         # two experts to a thread, none of them left over
    (513, 3, 1024, 700, True),          # nearly all of them left over
    (1000, 16, 512, 600, True),         # one to a thread, nobody's partner
    (64, 3, 8192, 3001, True),
])
def test_single_rank_dispatch_counts_and_claims(experts, topk, hidden, tokens, masked):
    import hcomm_b200 as hb
    from hcomm_b200.ops.moe import MoeExchange, quantize_e4m3_1x128
    torch.cuda.set_device(0)
    comm = hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=8)
    moe = MoeExchange(comm, experts, topk, hidden, tokens, capacity_factor=1.0)
    try:
        g = torch.Generator(device="cuda").manual_seed(tokens)
        x = torch.randn(tokens, hidden, device="cuda", generator=g).to(torch.bfloat16)
        idx = torch.rand(tokens, experts, device="cuda", generator=g).topk(topk, dim=1).indices.to(torch.int32).contiguous()
        if masked:
            idx[torch.rand(tokens, topk, device="cuda", generator=g) < 0.2] = -1
        rec = moe.dispatch(x, idx)
        flat = idx.flatten().long()
        kept = flat >= 0
        n = int(kept.sum())
        assert rec.num_rows == n and moe.overflow() == 0
        counts = torch.bincount(flat[kept], minlength=experts)
        assert torch.equal(rec.expert_offsets[1:].long(), counts.cumsum(0)) and int(rec.expert_offsets[0]) == 0
        at = rec.origin[:n]
        assert torch.equal(at.sort().values, kept.nonzero().flatten())
        assert bool((flat[at].diff() >= 0).all())
        q, scale = quantize_e4m3_1x128(x)
        assert torch.equal(rec.rows[:n].view(torch.uint8), q.view(torch.uint8)[at // topk]) and torch.equal(rec.scales[:n], scale[at // topk])
        assert torch.equal(moe.sent.flatten()[:tokens * topk] != 0, kept)
    finally:
        moe.destroy()
        comm.destroy()
