"""The measured work of the framework on one GPU: what a user's program asks of it through its public entry points.

    listed()              the cases, plain dicts
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what a program holds before the call (inputs, weights, workspaces)
    run(state)            one pass
    work(case)            bytes and operations that a pass cannot do without
    tolerance(case)       how far another correct implementation may be off
    exact(case, seed)     the same outputs in 64 bits by plain torch

Multi-rank paths (tensor-parallel block, collectives) run with all ranks on one device, one launch per call, as
``xccl_b200.ops`` offers it for a machine with a single GPU.
"""
import math

import torch

from xccl_b200.models.tp_mlp import TpMlp, TpMlpFp8
from xccl_b200.ops import gemm
from xccl_b200.ops.emu import EmuWorld
from xccl_b200.ops.moe import MoeWorkspace

BF16, F32, F64, F8 = torch.bfloat16, torch.float32, torch.float64, torch.float8_e4m3fn
DTYPES = {"f32": F32, "bf16": BF16}


def listed():
    return [
        # A projection while decoding a small batch: 16 tokens against a square 8192 matrix, bound by reading the weights.
        {"name": "gemm_decode", "kind": "gemm", "m": 16, "n": 8192, "k": 8192},
        # A product whose three sizes fit no tile: prompts of odd length, a vocabulary or head count that is not a power of two.
        {"name": "gemm_ragged", "kind": "gemm", "m": 1000, "n": 3592, "k": 2056},
        # The gate and up projections of one eighth of the 8192 x 28672 block for a prompt of 2048 tokens.
        {"name": "swiglu_shard", "kind": "swiglu", "m": 2048, "f": 3584, "k": 8192},
        # Block-scaled fp8 projection while decoding.
        {"name": "fp8_decode", "kind": "fp8", "m": 64, "n": 7168, "k": 8192},
        # Block-scaled fp8 projection of a long prompt.
        {"name": "fp8_prefill", "kind": "fp8", "m": 4096, "n": 8192, "k": 7168},
        # The whole MLP block while decoding: 128 tokens, 1.4 GB of weights.
        {"name": "mlp_decode", "kind": "mlp", "tokens": 128, "hidden": 8192, "ffn": 28672, "tp": 1, "fp8": False},
        # The benchmark's block: 8192 tokens, hidden 8192, FFN 28672.
        {"name": "mlp_prefill", "kind": "mlp", "tokens": 8192, "hidden": 8192, "ffn": 28672, "tp": 1, "fp8": False},
        # The same block in block-scaled fp8 for a prompt of 4096 tokens.
        {"name": "mlp_fp8_prefill", "kind": "mlp", "tokens": 4096, "hidden": 8192, "ffn": 28672, "tp": 1, "fp8": True},
        # The block over four ranks: allgather -> GEMM and GEMM -> reduce-scatter.
        {"name": "mlp_four_ranks", "kind": "mlp", "tokens": 2048, "hidden": 4096, "ffn": 14336, "tp": 4, "fp8": False},
        # Expert dispatch and combine while decoding: 256 experts, 8 of them per token.
        {"name": "moe_decode", "kind": "moe", "tokens": 128, "hidden": 7168, "experts": 256, "topk": 8, "ranks": 1},
        # The same for a prompt of 4096 tokens, the MoE benchmark's sizes.
        {"name": "moe_prefill", "kind": "moe", "tokens": 4096, "hidden": 7168, "experts": 256, "topk": 8, "ranks": 1},
        # Gradient bucket of 16 MiB averaged over eight ranks.
        {"name": "allreduce_bucket", "kind": "coll", "op": "allreduce", "ranks": 8, "count": 4 << 20, "dtype": "f32"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _up(v, step, lo, hi):
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "swiglu", "fp8", "fp8", "mlp", "mlp", "moe", "moe", "coll"])
    if kind == "gemm":   # any number of rows; the other two sizes in steps of 8
        return {"kind": kind, "m": int(_log(rng, 1, 8192)), "n": _up(_log(rng, 256, 8192), 8, 256, 8192),
                "k": _up(_log(rng, 256, 8192), 8, 256, 8192)}
    if kind == "swiglu":
        return {"kind": kind, "m": int(_log(rng, 1, 8192)), "f": _up(_log(rng, 256, 7168), 128, 256, 7168),
                "k": _up(_log(rng, 512, 8192), 8, 512, 8192)}
    if kind == "fp8":
        return {"kind": kind, "m": int(_log(rng, 1, 8192)), "n": _up(_log(rng, 256, 8192), 128, 256, 8192),
                "k": _up(_log(rng, 512, 8192), 128, 512, 8192)}
    if kind == "mlp":    # 128-row blocks per rank
        tp, fp8 = rng.choice([1, 1, 2, 4]), rng.random() < 0.4
        return {"kind": kind, "tokens": _up(_log(rng, 128, 4096), 128 * tp, 128 * tp, 4096),
                "hidden": _up(_log(rng, 1024, 8192), 128, 1024, 8192),
                "ffn": _up(_log(rng, 2048, 14336), 128 * tp, 2048, 14336), "tp": tp, "fp8": fp8}
    if kind == "moe":
        ranks = rng.choice([1, 1, 2, 4])
        return {"kind": kind, "tokens": int(_log(rng, 16, 4096 // ranks)), "hidden": _up(_log(rng, 1024, 7168), 8, 1024, 7168),
                "experts": rng.choice([16, 64, 128, 256]), "topk": rng.choice([2, 4, 6, 8]), "ranks": ranks}
    op = rng.choice(["allreduce", "allreduce", "reduce_scatter", "allgather", "alltoall"])
    ranks = rng.choice([2, 4, 8])
    return {"kind": kind, "op": op, "ranks": ranks, "count": max(ranks, int(_log(rng, 256, 4 << 20)) // ranks * ranks),
            "dtype": rng.choice(["f32", "bf16"])}


# ---------------------------------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, scale=1.0, dtype=BF16):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _linear_inputs(case, seed):
    """Activations of unit size whose rows differ in scale, and weights of 0.02 as in the block's initialisation."""
    g = _gen(seed)
    rows = case["f"] if case["kind"] == "swiglu" else case["n"]
    x = _randn(g, case["m"], case["k"], dtype=F32) * (0.5 + torch.rand(case["m"], 1, device="cuda", generator=g))
    return [x.to(BF16)] + [_randn(g, rows, case["k"], scale=0.02) for _ in range(2 if case["kind"] == "swiglu" else 1)]


def _mlp_inputs(case, seed):
    """x [tokens, hidden] and per rank (gate, up, down)."""
    g = _gen(seed)
    tp, hid, f = case["tp"], case["hidden"], case["ffn"] // case["tp"]
    x = _randn(g, case["tokens"], hid)
    return x, [(_randn(g, f, hid, scale=0.02), _randn(g, f, hid, scale=0.02), _randn(g, hid, f, scale=0.02)) for _ in range(tp)]


def _moe_inputs(case, seed):
    """Per rank: token rows, distinct experts per token, their probabilities as gate weights (not renormalised)."""
    g = _gen(seed)
    t, h, e, k = case["tokens"], case["hidden"], case["experts"], case["topk"]
    out = []
    for _ in range(case["ranks"]):
        logits = torch.randn(t, e, device="cuda", generator=g)
        top = logits.topk(k, dim=-1)
        gates = torch.softmax(logits, -1).gather(1, top.indices)
        out.append((_randn(g, t, h), top.indices.to(torch.int32).contiguous(), gates.contiguous()))
    return out


def _coll_inputs(case, seed):
    g = _gen(seed)
    return [_randn(g, case["count"], dtype=DTYPES[case["dtype"]]) for _ in range(case["ranks"])]


def _moe_capacity(case):
    rows = case["tokens"] * case["topk"]
    return case["ranks"] * rows if case["ranks"] == 1 else min(case["ranks"] * rows, 2 * rows + 64 * case["topk"])


class _State:
    """Inputs, outputs and the handle a program keeps; the handle is closed with the state."""

    def __init__(self, kind, handle=None, **kw):
        self.kind, self.handle = kind, handle
        self.__dict__.update(kw)

    def __del__(self):
        if self.handle is not None:
            self.handle.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        a, b = _linear_inputs(case, seed)
        return _State(kind, a=a, b=b, out=torch.empty(case["m"], case["n"], dtype=BF16, device="cuda"))
    if kind == "swiglu":
        a, wg, wu = _linear_inputs(case, seed)
        return _State(kind, a=a, wg=wg, wu=wu, out=torch.empty(case["m"], case["f"], dtype=BF16, device="cuda"))
    if kind == "fp8":
        a, b = _linear_inputs(case, seed)
        a8, sa = gemm.quantize_act_1x128(a)
        b8, sb = gemm.quantize_weight_128x128(b)
        return _State(kind, a=a8, sa=sa, b=b8, sb=sb, out=torch.empty(case["m"], case["n"], dtype=BF16, device="cuda"))
    if kind == "mlp":
        x, weights = _mlp_inputs(case, seed)
        cls = TpMlpFp8 if case["fp8"] else TpMlp
        mlp = cls(case["tokens"], case["hidden"], case["ffn"], tp=case["tp"])
        for i, ws in enumerate(weights):
            for name, w in zip(("gate", "up", "down"), ws):
                getattr(mlp, "w_" + name)[i].copy_(w)
                if case["fp8"]:
                    q, s = gemm.quantize_weight_128x128(w)
                    getattr(mlp, "w_%s8" % name)[i].copy_(q)
                    getattr(mlp, "s_" + name)[i].copy_(s)
        return _State(kind, mlp, x=[c.contiguous() for c in x.chunk(case["tp"], 0)])
    if kind == "moe":
        ins = _moe_inputs(case, seed)
        ws = MoeWorkspace(case["tokens"], case["hidden"], case["experts"], case["topk"], emu_ranks=case["ranks"],
                          cap_rows=_moe_capacity(case))
        ranks = range(case["ranks"])
        return _State(kind, ws, x=[i[0] for i in ins], ids=[i[1] for i in ins], gates=[i[2] for i in ins],
                      recv=[ws.recv(r) for r in ranks], expert_out=[ws.expert_out(r) for r in ranks],
                      rows=[ws.expert_rows(r) for r in ranks], out=[torch.empty_like(i[0]) for i in ins])
    src = _coll_inputs(case, seed)
    n, count = case["ranks"], case["count"]
    size = {"allreduce": count, "reduce_scatter": count // n, "allgather": count * n, "alltoall": count}[case["op"]]
    return _State(kind, EmuWorld(n, 64 << 20), op=case["op"], src=src, ranks=n,
                  dst=[torch.empty(size, dtype=s.dtype, device="cuda") for s in src])


def run(state):
    kind = state.kind
    if kind == "gemm":
        return gemm.gemm_bf16(state.a, state.b, state.out)
    if kind == "swiglu":
        return gemm.gemm_swiglu(state.a, state.wg, state.wu, state.out)
    if kind == "fp8":
        return gemm.gemm_fp8_blockscaled(state.a, state.sa, state.b, state.sb, state.out)
    if kind == "mlp":
        return state.handle.forward(state.x)
    if kind == "moe":
        # the experts hand their rows through unchanged, so that the all-to-all is what is measured
        state.handle.dispatch(state.x, state.ids)
        for dst, src in zip(state.expert_out, state.recv):
            dst.copy_(src)
        state.handle.combine(state.ids, state.gates, state.out)
        return {"out": state.out, "rows": state.rows}
    if state.op == "allreduce":
        state.handle.allreduce(state.src, state.dst, scale=1.0 / state.ranks)
    else:
        getattr(state.handle, state.op)(state.src, state.dst)
    return state.dst


def work(case):
    kind = case["kind"]
    if kind in ("gemm", "fp8"):
        m, n, k = case["m"], case["n"], case["k"]
        es = 2 if kind == "gemm" else 1
        scales = 0 if kind == "gemm" else 4 * (m * (k // 128) + (n // 128) * (k // 128))
        return {"bytes": es * (m * k + n * k) + scales + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "swiglu":
        m, f, k = case["m"], case["f"], case["k"]
        return {"bytes": 2 * (m * k + 2 * f * k + m * f), "flops": 4 * m * f * k}
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        es = 1 if case["fp8"] else 2
        return {"bytes": 2 * t * h + es * 3 * h * f + 2 * t * h, "flops": 6 * t * h * f}
    if kind == "moe":
        t, h, k = case["tokens"] * case["ranks"], case["hidden"], case["topk"]
        moved = _moe_capacity(case) * case["ranks"] * h * 2       # the experts' pass reads and writes the whole buffers
        return {"bytes": 2 * t * h + 2 * t * k * h + 2 * moved + 2 * t * k * h + 2 * t * h + 8 * t * k, "flops": 2 * t * k * h}
    es = 4 if case["dtype"] == "f32" else 2
    n, size = case["ranks"], case["count"] * (4 if case["dtype"] == "f32" else 2)
    if case["op"] == "allreduce":
        return {"bytes": 2 * n * size, "flops": n * case["count"]}
    if case["op"] == "reduce_scatter":
        return {"bytes": n * size + size, "flops": n * case["count"]}
    if case["op"] == "allgather":
        return {"bytes": n * size + n * n * size, "flops": 0}
    return {"bytes": 2 * n * case["count"] * es, "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "coll":
        if case["op"] in ("allgather", "alltoall"):
            return "exact"
        # sums of at most eight values in 32 bits, rounded once more where the buffers are bf16
        return {"rel": 1e-6} if case["dtype"] == "f32" else {"rel": 5e-3}
    if kind == "mlp" and case["fp8"]:
        # an intermediate value that falls on the other side of a rounding step moves by one e4m3 step (2^-3 of it);
        # measured against the 64-bit values with the same quantisation steps: 1.7e-2
        return {"rel": 2e-2}
    # bf16 outputs of 32-bit sums: half a unit in the last place is 2^-9 of the value, for either side
    return {"rel": 5e-3}


# ---------------------------------------------------------------------------------------------- 64-bit values

def _quant_rows(v):
    """e4m3 values and the scales (largest magnitude of 128 columns over 448) of a matrix, as 64-bit products."""
    r, c = v.shape
    b = v.to(F64).view(r, c // 128, 128)
    s = (b.abs().amax(-1, keepdim=True).clamp_min(1e-12).to(F32) / 448.0)
    return ((b * (1.0 / s)).to(F32).to(F8).to(F64) * s.to(F64)).view(r, c)


def _quant_acts(v):
    r, c = v.shape
    b = v.to(F32).view(r, c // 128, 128)
    s = b.abs().amax(-1, keepdim=True).clamp_min(1e-12) / 448.0
    return ((b / s).to(F8).to(F64) * s.to(F64)).view(r, c)


def _quant_weight(w):
    n, k = w.shape
    b = w.to(F32).view(n // 128, 128, k // 128, 128)
    s = b.abs().amax((1, 3), keepdim=True).clamp_min(1e-12) / 448.0
    return ((b / s).to(F8).to(F64) * s.to(F64)).view(n, k)


def _silu_mul(g, u):
    return g / (1.0 + torch.exp(-g)) * u


def exact(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        a, b = _linear_inputs(case, seed)
        return a.to(F64) @ b.to(F64).t()
    if kind == "swiglu":
        a, wg, wu = _linear_inputs(case, seed)
        a = a.to(F64)
        return _silu_mul(a @ wg.to(F64).t(), a @ wu.to(F64).t())
    if kind == "fp8":
        a, b = _linear_inputs(case, seed)
        return _quant_acts(a) @ _quant_weight(b).t()
    if kind == "mlp":
        x, weights = _mlp_inputs(case, seed)
        y = torch.zeros(case["tokens"], case["hidden"], dtype=F64, device="cuda")
        x = _quant_rows(x.to(F32)) if case["fp8"] else x.to(F64)
        for wg, wu, wd in weights:
            up = _quant_weight if case["fp8"] else (lambda w: w.to(F64))
            h = _silu_mul(x @ up(wg).t(), x @ up(wu).t())
            y += (_quant_rows(h) if case["fp8"] else h) @ up(wd).t()
        return list(y.chunk(case["tp"], 0))
    if kind == "moe":
        ins = _moe_inputs(case, seed)
        el = case["experts"] // case["ranks"]
        counts = sum(torch.bincount(i[1].flatten().long(), minlength=case["experts"]) for i in ins)
        rows = []
        for r in range(case["ranks"]):
            mine = counts[r * el:(r + 1) * el]
            rows.append(torch.cat([mine, mine.sum()[None]]))
        return {"out": [i[0].to(F64) * i[2].to(F64).sum(-1, keepdim=True) for i in ins], "rows": rows}
    src = _coll_inputs(case, seed)
    n = case["ranks"]
    if case["op"] == "allgather":
        return [torch.cat(src).to(F64) for _ in range(n)]
    if case["op"] == "alltoall":
        parts = [s.to(F64).chunk(n) for s in src]
        return [torch.cat([parts[s][d] for s in range(n)]) for d in range(n)]
    total = sum(s.to(F64) for s in src)
    if case["op"] == "allreduce":
        return [total / n for _ in range(n)]
    return list(total.chunk(n))
