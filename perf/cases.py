"""The calls that one GPU makes through the library's public entry points, over the sizes that they are made at.

Six kinds of work:

``linear``   ``ops.gemm.gemm_bf16``: one projection, ``a @ b.T``
``mlp``      ``parallel.tp.TensorParallelMlp``: up and down projection of a decoder layer, from one decoded token to a prefill
``moe``      ``ops.moe.MoeExchange``: dispatch (routing, fp8 quantisation), the experts' step, combine (gate-weighted sum)
``dispatch`` the first half alone; the rows of an expert come in no fixed order, so they are put in that of the tokens
``combine``  the second half alone, on a routing that was dispatched before
``coll``     one operator of a communicator (a data-parallel bucket, a small reduction, gathers and exchanges)

Widths are those of ``models.llama.CONFIGS``, of one rank's share of them under tensor parallelism over eight ranks, and of
the expert-parallel benchmark (256 experts, 8 per token, hidden 7168).
"""
import functools
import weakref

import torch

import hcomm_b200 as hb
from hcomm_b200.ops.gemm import gemm_bf16
from hcomm_b200.ops.moe import MoeExchange
from hcomm_b200.parallel.tp import TensorParallelMlp

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16, "int32": torch.int32}

# (hidden, intermediate) of the feed-forward layer: llama3_70b, one of eight ranks' share of it, llama3_8b, small
MLPS = [(8192, 28672), (8192, 3584), (4096, 14336), (1024, 4096)]
# (out features, in features) of single projections: q / o, k / v, the vocabulary of llama3_8b and of small, odd ones
LINEARS = [(4096, 4096), (1024, 4096), (8192, 8192), (128256, 4096), (32000, 1024), (3584, 1000), (136, 72), (5000, 2056)]


def listed():
    return [
        # the smallest call: nothing but a launch and its latency
        {"name": "linear-tiny", "kind": "linear", "m": 200, "n": 136, "k": 72, "pitch": 0},
        # logits of the last position of 33 sequences: rows of a [batch, seq, hidden] tensor, so their pitch is 16 rows wide
        {"name": "linear-logits", "kind": "linear", "m": 33, "n": 128256, "k": 4096, "pitch": 16},
        # decoding with a batch of 16: every weight is read for a handful of rows
        {"name": "mlp-decode-16", "kind": "mlp", "tokens": 16, "hidden": 8192, "inter": 28672},
        # the same layer split over eight ranks, a batch of 96
        {"name": "mlp-share-96", "kind": "mlp", "tokens": 96, "hidden": 8192, "inter": 3584},
        # one chunk of a prefill, as long as the prompt's rest happens to be
        {"name": "mlp-chunk-777", "kind": "mlp", "tokens": 777, "hidden": 4096, "inter": 14336},
        # packed prompts of no round length on one rank's share
        {"name": "mlp-share-5003", "kind": "mlp", "tokens": 5003, "hidden": 8192, "inter": 3584},
        # the benchmark's step: 8192 tokens through the whole layer
        {"name": "mlp-prefill-8192", "kind": "mlp", "tokens": 8192, "hidden": 8192, "inter": 28672},
        # experts while decoding: there and back for a few tokens
        {"name": "moe-decode-64", "kind": "moe", "tokens": 64, "hidden": 7168, "experts": 256, "topk": 8, "masked": False},
        # every token of a prefill to its eight experts
        {"name": "dispatch-prefill-4096", "kind": "dispatch", "tokens": 4096, "hidden": 7168, "experts": 256, "topk": 8, "masked": False},
        # expert outputs back to an odd number of tokens, some choices masked
        {"name": "combine-3001", "kind": "combine", "tokens": 3001, "hidden": 7168, "experts": 256, "topk": 8, "masked": True},
        # one bucket of gradients, averaged over eight accumulated steps; parameters do not add up to a round number
        {"name": "coll-bucket", "kind": "coll", "op": "all_reduce_scaled", "dtype": "bf16", "count": 33361921, "offset": 0},
        # a loss or a norm shared by all ranks: a reduction of a few KB
        {"name": "coll-small", "kind": "coll", "op": "all_reduce", "dtype": "fp32", "count": 2048, "offset": 0},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread evenly over their logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["linear"] * 3 + ["mlp"] * 4 + ["moe", "dispatch", "combine"] + ["coll"] * 2)
    if kind == "linear":
        n, k = rng.choice(LINEARS)
        return {"kind": kind, "m": _log(rng, 1, 4096 if n < 100000 else 256), "n": n, "k": k, "pitch": rng.choice([0, 0, 2])}
    if kind == "mlp":
        hidden, inter = rng.choice(MLPS)
        return {"kind": kind, "tokens": _log(rng, 1, 8192), "hidden": hidden, "inter": inter}
    if kind in ("moe", "dispatch", "combine"):
        hidden = rng.choice([512, 2048, 4096, 7168, 8192])
        experts, topk = rng.choice([(8, 2), (64, 6), (128, 4), (256, 8)])
        tokens = _log(rng, 1, 256 if kind == "moe" else 4096)
        return {"kind": kind, "tokens": tokens, "hidden": hidden, "experts": experts, "topk": topk, "masked": kind != "dispatch" and rng.random() < 0.3}
    op = rng.choice(["all_reduce", "all_reduce_scaled", "all_gather", "reduce_scatter", "all_to_all", "all_to_all_v"])
    dtype = rng.choice(["fp32", "bf16", "fp16"] if op == "all_reduce_scaled" else ["fp32", "bf16", "fp16", "int32"])
    count = _log(rng, 64, 1 << 26) | rng.randrange(2)
    return {"kind": kind, "op": op, "dtype": dtype, "count": count, "offset": rng.choice([0, 0, 0, 3])}


@functools.lru_cache(maxsize=None)
def _communicator():
    """The program's one communicator."""
    return hb.Communicator(1, hb.get_root_info(), 0, buffer_mb=64)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def _normal(g, rows, cols, std):
    return (torch.randn(rows, cols, device="cuda", generator=g) * std).to(torch.bfloat16)


class State:
    """What a program holds between calls."""


def _linear_inputs(case, seed):
    g = _generator(seed)
    m, n, k, pitch = case["m"], case["n"], case["k"], case["pitch"]
    if pitch:
        a = _normal(g, m * pitch, k, 1.0).view(m, pitch, k)[:, -1]      # the last position of every sequence
    else:
        a = _normal(g, m, k, 1.0)
    return a, _normal(g, n, k, 0.02)


def _mlp_inputs(case, seed):
    g = _generator(seed)
    x = _normal(g, case["tokens"], case["hidden"], 1.0)
    w_up = _normal(g, case["inter"], case["hidden"], 0.02)
    w_down = _normal(g, case["hidden"], case["inter"], 0.02)
    return x, w_up, w_down


def _moe_inputs(case, seed):
    """Router logits are N(0, 1): the choices of a token are the largest, the gates their softmax."""
    g = _generator(seed)
    t, e, k = case["tokens"], case["experts"], case["topk"]
    x = _normal(g, t, case["hidden"], 1.0)
    top = torch.randn(t, e, device="cuda", generator=g).topk(k, dim=1)
    idx = top.indices.to(torch.int32).contiguous()
    if case["masked"]:          # padding tokens and choices that the router took back
        idx[torch.rand(t, k, device="cuda", generator=g) < 0.1] = -1
    return x, idx, torch.softmax(top.values, dim=1).contiguous()


def _coll_inputs(case, seed):
    g = _generator(seed)
    n, off = case["count"], case["offset"]
    dt = DTYPES[case["dtype"]]
    if dt == torch.int32:
        full = torch.randint(-1000, 1000, (n + off,), device="cuda", generator=g, dtype=dt)
    else:
        full = torch.randn(n + off, device="cuda", generator=g).to(dt)
    return full[off:]           # a view into a flat buffer: not every slice of one starts on 16 bytes


def _exchange(s, case):
    moe = MoeExchange(_communicator(), case["experts"], case["topk"], case["hidden"], case["tokens"], capacity_factor=1.0)
    weakref.finalize(s, moe.destroy)
    return moe


def _experts(rec, y):
    """Stands for the experts: every received row back in bf16, in the order it was received in, with its scales in bf16."""
    n, h = y.shape
    y.copy_(rec.rows[:n])
    y.view(n, -1, 128).mul_(rec.scales[:n].to(torch.bfloat16).unsqueeze(-1))


def prepare(case, seed):
    s = State()
    s.kind, s.case = case["kind"], case
    if s.kind == "linear":
        s.a, s.b = _linear_inputs(case, seed)
    elif s.kind == "mlp":
        s.x, w_up, w_down = _mlp_inputs(case, seed)
        s.mlp = TensorParallelMlp(_communicator(), case["hidden"], case["inter"], w_up=w_up, w_down=w_down)
    elif s.kind in ("moe", "dispatch", "combine"):
        s.x, s.idx, s.gates = _moe_inputs(case, seed)
        s.moe = _exchange(s, case)
        n, h = case["tokens"] * case["topk"], case["hidden"]
        if s.kind == "dispatch":
            s.rows = torch.zeros(n, h, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
            s.scales = torch.zeros(n, h // 128, device="cuda")
        else:
            s.y = torch.zeros(n, h, dtype=torch.bfloat16, device="cuda")
        if s.kind == "combine":
            _experts(s.moe.dispatch(s.x, s.idx), s.y)
    else:
        s.comm = _communicator()
        s.x = _coll_inputs(case, seed)
        s.out = torch.empty_like(s.x)
    return s


def run(s):
    if s.kind == "linear":
        return gemm_bf16(s.a, s.b)
    if s.kind == "mlp":
        return s.mlp(s.x)
    if s.kind == "moe":
        _experts(s.moe.dispatch(s.x, s.idx), s.y)
        return s.moe.combine(s.y, s.gates)
    if s.kind == "dispatch":
        rec, n = s.moe.dispatch(s.x, s.idx), s.rows.shape[0]
        at = rec.origin[:n]                 # token * topk + choice: with one rank there is no other part
        s.rows.view(torch.int64).index_copy_(0, at, rec.rows[:n].view(torch.int64))
        s.scales.index_copy_(0, at, rec.scales[:n])
        return {"rows": s.rows, "scales": s.scales, "offsets": rec.expert_offsets.clone()}     # the exchange's own buffer goes with it
    if s.kind == "combine":
        return s.moe.combine(s.y, s.gates)
    op, n = s.case["op"], s.case["count"]
    if op == "all_reduce_scaled":
        return s.comm.all_reduce_scaled(s.x, s.out, 0.125)
    if op == "all_to_all_v":
        return s.comm.all_to_all_v(s.x, [n], [0], s.out, [n], [0])
    return getattr(s.comm, op)(s.x, s.out)


def work(case):
    """Operands once in, results once out.  ``moe`` hands rows to the experts and takes theirs back, so those count as well,
    and ``dispatch`` reads them for their order."""
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    if kind == "mlp":
        t, h, i = case["tokens"], case["hidden"], case["inter"]
        return {"bytes": 2 * (2 * t * h + 2 * h * i), "flops": 4 * t * h * i}
    if kind in ("moe", "dispatch", "combine"):
        t, h, k = case["tokens"], case["hidden"], case["topk"]
        combine = 2 * t * k * h + 2 * t * h + 4 * t * k
        if kind == "combine":
            return {"bytes": combine, "flops": 2 * t * k * h}
        row = h + h // 32                                       # fp8 values and their scales
        dispatch = 2 * t * h + 4 * t * k + t * k * (row + 8)
        if kind == "dispatch":
            return {"bytes": dispatch + 2 * t * k * row, "flops": 0}
        return {"bytes": dispatch + t * k * (row + 2 * h) + combine, "flops": 2 * t * k * h}
    return {"bytes": 2 * case["count"] * DTYPES[case["dtype"]].itemsize, "flops": 0}


def tolerance(case):
    """bf16 results of 32-bit sums in another order: where a sum falls next to a rounding boundary the result moves by one
    step of bf16, and in ``mlp`` the hidden values that moved so are summed once more.  Rows and copies stay the same bytes."""
    if case["kind"] in ("linear", "mlp"):
        return {"rel": 5e-3, "max": 3e-2}
    if case["kind"] in ("moe", "combine"):
        return {"rel": 5e-3, "max": 2e-2}
    return "exact"


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        a, b = _linear_inputs(case, seed)
        return a.double() @ b.double().t()
    if kind == "mlp":
        x, w_up, w_down = _mlp_inputs(case, seed)
        return (x.double() @ w_up.double().t()) @ w_down.double().t()
    if kind in ("moe", "dispatch", "combine"):
        x, idx, gates = _moe_inputs(case, seed)
        t, h = x.shape
        blocks = x.float().view(t, h // 128, 128)
        scale = blocks.abs().amax(dim=-1, keepdim=True).clamp_min(1e-4)
        scale = scale / torch.full_like(scale, 448.0)
        q = (blocks / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
        if kind == "dispatch":
            k = case["topk"]
            return {"rows": q.double().view(t, h).repeat_interleave(k, 0), "scales": scale.double().view(t, -1).repeat_interleave(k, 0), "offsets": None}
        rows = (q.double() * scale.to(torch.bfloat16).double()).view(t, h)
        kept = torch.where((idx >= 0) & (idx < case["experts"]), gates.double(), 0.0)
        return rows * kept.sum(dim=1, keepdim=True)
    x = _coll_inputs(case, seed)
    return x.double() * 0.125 if case["op"] == "all_reduce_scaled" else (x.double() if x.is_floating_point() else x)
