"""What this framework is used for, as timed cases: bytecode programs run through its public entry points.

A case names a program family (``kind``) and its sizes. Every family is a program that a user has the framework run: element-wise
kernels and row reductions as the torch.compile backend lowers them, the hand-written head-wise normalisation in bfloat16, the
small-matrix programs, a compiled graph of several launches, and batches of candidate programs of a superoptimizer. The programs
are written with the framework's own emitters (or, for the 4x4 inverse, take the recorded instruction stream, which does not depend
on the batch size), so that every size of a family can be built.
"""
import functools
import math

import numpy as np
import torch

from gint_b200 import BaseExecutableProgram, ProgramData, ProgramTensorInfo, bytecode, cdiv, get_executor
from gint_b200 import opcodes as O
from gint_b200.feeder import BatchRunner
from gint_b200.host import frontend as F
from gint_b200.host.executor import _convert_arg
from gint_b200.programs import recorded

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}
EPS = 1e-6


# ---------------------------------------------------------------------------------------------- programs

@bytecode
def add(out, a, b, REGW, WARP):
    """out = a + b, one tile of 128 values per logical program."""
    n, = a.shape
    tile = REGW * WARP
    out, a, b = [F.make_block_1d(t, n, t.strides[0], cdiv(n, tile), tile) for t in (out, a, b)]
    F.fldg_1d(0, a)
    F.fldg_1d(0, b)
    F.fadd()
    F.fstg_1d(0, out)
    F.halt()


@bytecode
def gated_silu(out, a, b, REGW, WARP, dtype="f32"):
    """out = a * sigmoid(a) * b, four tiles per logical program."""
    n, = a.shape
    load = {"f32": F.fldg_1d, "f16": F.fldg_1d_f16, "bf16": F.fldg_1d_bf16}[dtype]
    store = {"f32": F.fstg_1d, "f16": F.fstg_1d_f16, "bf16": F.fstg_1d_bf16}[dtype]
    tile = REGW * WARP
    block = 4 * tile
    out, a, b = [F.make_block_1d(t, n, t.strides[0], cdiv(n, block), block) for t in (out, a, b)]
    for off in range(0, block, tile):
        load(off, a)
        F.dup()
        F.fneg()
        F.fexp()
        F.faddimm(1.0)
        F.frdiv()
        load(off, b)
        F.fmul()
        store(off, out)
    F.halt()


def row_scale(x, n, tile):
    """Leaves rsqrt(mean(x^2) + eps) of the row on the stack, in every lane."""
    for off in range(0, n, tile):
        F.fldg_1d(off, x)
        F.fldg_1d(off, x)
        F.fmul()
        if off:
            F.fadd()
    row_total()
    F.fmulimm(1.0 / n)
    F.faddimm(EPS)
    F.frsqrt()


def row_total():
    """Adds the top of the stack up over the lanes and the four values of each."""
    F.warp_allreduce_fsum()
    F.dup()
    F.fperm_w(2, 3, 0, 1)
    F.fadd()
    F.dup()
    F.fperm_w(1, 0, 3, 2)
    F.fadd()


def row_block(t, rows, n, stride):
    return F.make_block_1d(t, n, 1, 1, n, [stride], [rows])


@bytecode
def rmsnorm(x, w, out, REGW, WARP):
    """out = x * rsqrt(mean(x^2) + eps) * w, one row per logical program."""
    rows, n = x.shape
    tile = REGW * WARP
    xb, wb, ob = row_block(x, rows, n, n), row_block(w, rows, n, 0), row_block(out, rows, n, n)
    row_scale(xb, n, tile)
    for off in range(0, n, tile):
        F.dup()
        F.fldg_1d(off, xb)
        F.swap()
        F.fmul()
        F.fldg_1d(off, wb)
        F.fmul()
        F.fstg_1d(off, ob)
    F.pop()
    F.halt()


@bytecode
def rmsnorm_silu_residual(z, x, w, g, REGW, WARP):
    """z = silu(rmsnorm(g) * w) + x, one row per logical program: the fused subgraph of the compiled graph."""
    rows, n = z.shape
    tile = REGW * WARP
    zb, xb, wb, gb = row_block(z, rows, n, n), row_block(x, rows, n, n), row_block(w, rows, n, 0), row_block(g, rows, n, n)
    row_scale(gb, n, tile)
    for off in range(0, n, tile):
        F.dup()
        F.fldg_1d(off, gb)
        F.swap()
        F.fmul()
        F.fldg_1d(off, wb)
        F.fmul()
        F.dup()
        F.fneg()
        F.fexp()
        F.faddimm(1.0)
        F.frdiv()
        F.fldg_1d(off, xb)
        F.fadd()
        F.fstg_1d(off, zb)
    F.pop()
    F.halt()


@bytecode
def row_sum(z, s, REGW, WARP):
    """s = z.sum(-1), one row per logical program: the second subgraph of the compiled graph."""
    rows, n = z.shape
    tile = REGW * WARP
    zb = F.make_block_2d(z, [n, rows], [1, n], [1, rows], [tile, 1])
    sb = F.make_block_2d(s, [1, rows], [1, 1], [1, rows], [1, 1])
    for off in range(0, n, tile):
        F.fldg_1d(off, zb)
        if off:
            F.fadd()
    row_total()
    F.fstg_1d(0, sb)
    F.halt()


@bytecode
def head_rmsnorm(x, y, w, REGW, WARP):
    """rmsnorm of bfloat16 heads, (batch, heads, tokens, dim) views of a (batch, tokens, heads, dim) tensor; four tokens per logical program."""
    B, NH, T, H = x.shape
    xb, yb = [F.make_block_2d(t, [H, T], [t.strides[-1], t.strides[-2]], [1, cdiv(T, REGW)], [0, REGW], [t.strides[0], t.strides[1]], [B, NH])
              for t in (x, y)]
    wb = F.make_block_2d(w, [H, T], [w.strides[-1], 0], [1, cdiv(T, REGW)], [0, REGW], [0, 0], [B, NH])
    F.fpush(0.0)
    for c in range(0, H, WARP):
        F.fldg_2dt_bf16(c, xb)
        F.dup()
        F.fma()
    F.warp_allreduce_fsum()
    F.fmaimm(1 / H, 1e-5)
    F.frsqrt()
    for c in range(0, H, WARP):
        F.dup()
        F.fldg_2dt_bf16(c, xb)
        F.fmul()
        F.fldg_2dt_bf16(c, wb)
        F.fmul()
        F.fstg_2dt_bf16(c, yb)
    F.halt()


def matrix_block(t, B):
    return F.make_block_2d(t, [B, 16], [16, 1], [cdiv(B, 32), 1], [32, 0])


@bytecode
def bmm4x4(a, b, c, REGW, WARP):
    """c = a @ b, one 4x4 matrix per lane."""
    B, _ = a.shape
    ab, bb, cb = matrix_block(a, B), matrix_block(b, B), matrix_block(c, B)
    for i in range(4):
        F.fldg_2dw(4 * i, ab)
        for k in range(4):
            F.dup_broadcast_w(k)
            F.fldg_2dw(4 * k, bb)
            F.fmul()
            F.swap()
        F.pop()
        F.fadd()
        F.fadd()
        F.fadd()
        F.fstg_2dw(4 * i, cb)
    F.halt()


class Inverse4x4(BaseExecutableProgram):
    """c = inv(a), one 4x4 matrix per lane: the recorded stream, with the descriptors of the batch that is passed."""

    def get_program(self, a, c):
        B, _ = a.shape
        info = ProgramTensorInfo(4, [], [], [B, 16], [16, 1], [cdiv(B, 32), 1], [32, 0])
        return ProgramData(recorded("inv4x4_b33").bytecode, [info, info])


inv4x4 = Inverse4x4()


# ---------------------------------------------------------------------------------------------- candidates of a superoptimizer

UNARY, BINARY = [O.FNeg, O.FRcp, O.FSqrt], [O.FAdd, O.FMul, O.FSub, O.FRSub, O.FGt, O.FLt]


def candidates(rng, count, body):
    """int32 [count, words]: load two inputs, `body` random stack-valid instructions, fold the stack, store; padded with Nops to one length."""
    slots = 2 + body + 6 + 2
    code = np.zeros((count, slots, 2), dtype=np.int32)
    code[:, :, 0] = O.Nop
    code[:, 0] = O.LoadGlobal1DF32, 0
    code[:, 1] = O.LoadGlobal1DF32, 1
    depth = np.full(count, 2)
    for k in range(2, 2 + body):
        pick = rng.random(count)
        imm = rng.standard_normal(count).astype(np.float32).view(np.int32)
        sel = rng.integers(0, 4, (count, 4)) << np.array([0, 8, 16, 24])
        op = np.where(pick < 0.15, O.FMulImm, np.where(pick < 0.25, O.FPermW, rng.choice(UNARY, count)))
        operand = np.where(op == O.FMulImm, imm, np.where(op == O.FPermW, sel.sum(1), 0))
        grow = (pick > 0.4) & (depth < 6)
        op = np.where(grow, np.where(pick < 0.55, O.LoadImm, O.Dup), op)
        operand = np.where(grow, np.where(pick < 0.55, imm, 0), operand)
        two = (pick > 0.65) & (depth >= 2)
        op = np.where(two, np.where(pick > 0.93, O.Swap, rng.choice(BINARY, count)), op)
        operand = np.where(two, 0, operand)
        depth = depth + np.where(two, np.where(op == O.Swap, 0, -1), grow.astype(int))
        code[:, k, 0], code[:, k, 1] = op, operand
    for k in range(2 + body, slots - 2):
        code[:, k, 0] = np.where(depth > 1, O.FAdd, O.Nop)
        depth = np.maximum(depth - 1, 1)
    code[:, slots - 2] = O.StoreGlobal1DF32, 2
    code[:, slots - 1] = O.Halt, 0
    return code.reshape(count, 2 * slots)


# ---------------------------------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest call: one launch of a few blocks, where host time and launch latency are everything
        {"name": "add_4096", "kind": "add", "n": 4096},
        # the benchmark's element-wise program (a + b over 2^20 values)
        {"name": "add_1m", "kind": "add", "n": 1048576},
        # a large flat tensor whose length is no multiple of anything
        {"name": "add_ragged_40m", "kind": "add", "n": 40000003},
        # an activation between two half-precision layers, of a length that fills no last tile
        {"name": "gated_silu_f16", "kind": "gated_silu", "n": 24000500, "dtype": "f16"},
        # the benchmark's headline: rows of 4096, whole tiles
        {"name": "rmsnorm_16384x4096", "kind": "rmsnorm", "rows": 16384, "n": 4096},
        # rows as they come: neither the row count nor the row length is round, rows start at odd addresses
        {"name": "rmsnorm_ragged_10007x2029", "kind": "rmsnorm", "rows": 10007, "n": 2029},
        # per-head normalisation of a bfloat16 projection, as in the repository's own test of it, at a training size
        {"name": "head_rmsnorm_bf16", "kind": "head_rmsnorm", "batch": 8, "tokens": 4096, "heads": 16, "dim": 128},
        # the benchmark's compiled graph, rows gathered in place: two launches
        {"name": "graph_gathered_65536x1024", "kind": "graph_gathered", "rows": 65536, "n": 1024},
        # the same graph at a serving size: a gather kernel and a prepared plan of two launches
        {"name": "graph_plan_96x1024", "kind": "graph_plan", "rows": 96, "n": 1024},
        # the benchmark's small-matrix programs at their full size
        {"name": "bmm4x4_4194304", "kind": "bmm4x4", "batch": 4194304},
        {"name": "inv4x4_4194304", "kind": "inv4x4", "batch": 4194304},
        # one generation of a superoptimizer's candidates: many short programs, each run once
        {"name": "candidates_4096", "kind": "candidates", "count": 4096, "body": 16},
    ]


def log_int(rng, lo, hi):
    """Spread over the logarithm of the range; half of the values odd, the others rounded to a multiple of a power of two."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5:
        return min(hi, max(lo, v | 1))
    grain = 2 ** rng.randint(1, 7)
    return min(hi, max(lo, v // grain * grain))


def draw(rng):
    kind = rng.choice(["add", "gated_silu", "rmsnorm", "rmsnorm", "head_rmsnorm", "graph_gathered", "graph_plan", "bmm4x4", "inv4x4", "candidates"])
    if kind == "add":
        return {"kind": kind, "n": log_int(rng, 1000, 80_000_000)}
    if kind == "gated_silu":
        return {"kind": kind, "n": log_int(rng, 4000, 60_000_000), "dtype": rng.choice(["f32", "f16", "bf16"])}
    if kind == "rmsnorm":
        n = log_int(rng, 129, 6000)
        return {"kind": kind, "rows": log_int(rng, 3, 80_000_000 // n), "n": n}
    if kind == "head_rmsnorm":
        heads, dim = rng.randint(1, 24), rng.choice([64, 80, 96, 128])
        tokens = log_int(rng, 12, 8192)
        return {"kind": kind, "batch": rng.randint(1, max(1, min(8, 100_000_000 // (heads * dim * tokens)))), "tokens": tokens, "heads": heads, "dim": dim}
    if kind in ("graph_gathered", "graph_plan"):
        n = log_int(rng, 256, 4096)
        return {"kind": kind, "rows": log_int(rng, 10, 50_000_000 // n), "n": n}
    if kind in ("bmm4x4", "inv4x4"):
        return {"kind": kind, "batch": log_int(rng, 33, 4_000_000)}
    return {"kind": kind, "count": log_int(rng, 100, 4096), "body": rng.randint(4, 24)}


# ---------------------------------------------------------------------------------------------- a pass

def inputs(case, seed):
    """The tensors of a case by role; made on the GPU from the seed."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    randn = functools.partial(torch.randn, generator=g, device="cuda")
    rand = functools.partial(torch.rand, generator=g, device="cuda")
    kind = case["kind"]
    if kind == "add":
        return {"out": torch.zeros(case["n"], device="cuda"), "a": randn(case["n"]), "b": randn(case["n"])}
    if kind == "gated_silu":
        dt = DTYPES[case["dtype"]]
        return {"out": torch.zeros(case["n"], dtype=dt, device="cuda"), "a": randn(case["n"]).to(dt), "b": randn(case["n"]).to(dt)}
    if kind == "rmsnorm":
        return {"x": randn(case["rows"], case["n"]), "w": 1.0 + 0.1 * randn(case["n"]), "out": torch.zeros(case["rows"], case["n"], device="cuda")}
    if kind == "head_rmsnorm":
        x = (randn(case["batch"], case["tokens"], case["heads"], case["dim"]) * 1.5 + 0.5).to(torch.bfloat16)
        return {"x": x.transpose(1, 2), "y": torch.zeros_like(x).transpose(1, 2), "w": rand(case["dim"]).to(torch.bfloat16)}
    if kind in ("graph_gathered", "graph_plan"):
        rows, n = case["rows"], case["n"]
        t = {"x": randn(rows, n), "idx": torch.randint(0, rows, (rows,), generator=g, device="cuda"), "w": 1.0 + 0.1 * randn(n),
             "z": torch.zeros(rows, n, device="cuda"), "s": torch.zeros(rows, device="cuda")}
        if kind == "graph_plan":
            t["g"] = torch.zeros(rows, n, device="cuda")
        return t
    if kind == "bmm4x4":
        return {"a": rand(case["batch"], 16) * 2 - 1, "b": rand(case["batch"], 16) * 2 - 1, "c": torch.zeros(case["batch"], 16, device="cuda")}
    if kind == "inv4x4":
        return {"a": rand(case["batch"], 16) * 2 - 1 + 4.0 * torch.eye(4, device="cuda").reshape(16), "c": torch.zeros(case["batch"], 16, device="cuda")}
    return {"a": rand(128) + 0.5, "b": rand(128) + 0.5, "out": torch.zeros(case["count"], 128, device="cuda")}


def prepare(case, seed):
    """The tensors, and what a program keeps beside them: converted arguments and plans for the compiled graphs, the runner of a candidate batch."""
    s = {"case": case, "t": inputs(case, seed)}
    t, kind = s["t"], case["kind"]
    if kind == "graph_gathered":
        s["args"] = {k: _convert_arg(v) for k, v in t.items() if k != "idx"}
        s["args"]["table"] = _convert_arg(t["x"])    # the same rows once more, read through the index
    elif kind == "graph_plan":
        s["plan"] = get_executor().build_plan([(rmsnorm_silu_residual, [t["z"], t["x"], t["w"], t["g"]], case["rows"]),
                                               (row_sum, [t["z"], t["s"]], case["rows"])])
    elif kind == "candidates":
        s["runner"] = BatchRunner(n_inputs=2, test_size=128)
        s["codes"] = candidates(np.random.default_rng(seed), case["count"], case["body"])
    return s


def run(s):
    case, t = s["case"], s["t"]
    kind = case["kind"]
    if kind == "add":
        add(t["out"], t["a"], t["b"], grid_dim=cdiv(case["n"], 128))
        return t["out"]
    if kind == "gated_silu":
        gated_silu(t["out"], t["a"], t["b"], grid_dim=cdiv(case["n"], 512), dtype=case["dtype"])
        return t["out"]
    if kind == "rmsnorm":
        rmsnorm(t["x"], t["w"], t["out"], grid_dim=case["rows"])
        return t["out"]
    if kind == "head_rmsnorm":
        head_rmsnorm(t["x"], t["y"], t["w"], grid_dim=case["batch"] * case["heads"] * cdiv(case["tokens"], 4))
        return t["y"]
    if kind == "bmm4x4":
        bmm4x4(t["a"], t["b"], t["c"], grid_dim=cdiv(case["batch"], 32))
        return t["c"]
    if kind == "inv4x4":
        inv4x4(t["a"], t["c"], grid_dim=cdiv(case["batch"], 32))
        return t["c"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "graph_gathered":
        ex, a = get_executor(), s["args"]
        ex.execute_gathered(rmsnorm_silu_residual, [a["z"], a["x"], a["w"], a["table"]], case["rows"], (3,), t["idx"], cuda_stream=stream)
        ex.execute(row_sum, [a["z"], a["s"]], case["rows"], cuda_stream=stream)
        return t["z"], t["s"]
    if kind == "graph_plan":
        torch.index_select(t["x"], 0, t["idx"], out=t["g"])
        s["plan"].run(stream)
        return t["z"], t["s"]
    return s["runner"].run(s["codes"], [t["a"], t["b"]], t["out"], cuda_stream=stream)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "add":
        return {"bytes": 12 * case["n"], "flops": case["n"]}
    if kind == "gated_silu":
        return {"bytes": 3 * SIZE[case["dtype"]] * case["n"], "flops": 5 * case["n"]}
    if kind == "rmsnorm":
        return {"bytes": 8 * case["rows"] * case["n"] + 4 * case["n"], "flops": 4 * case["rows"] * case["n"]}
    if kind == "head_rmsnorm":
        n = case["batch"] * case["tokens"] * case["heads"] * case["dim"]
        return {"bytes": 4 * n + 2 * case["dim"], "flops": 4 * n}
    if kind in ("graph_gathered", "graph_plan"):
        rows, n = case["rows"], case["n"]
        # the gathered rows and the residual rows read, z written; the index, the weights and the sums beside them
        return {"bytes": 12 * rows * n + 12 * rows + 4 * n, "flops": 11 * rows * n}
    if kind == "bmm4x4":
        return {"bytes": 192 * case["batch"], "flops": 112 * case["batch"]}
    if kind == "inv4x4":
        return {"bytes": 128 * case["batch"], "flops": 250 * case["batch"]}
    words = 2 * (case["body"] + 10)
    return {"bytes": case["count"] * (4 * words + 512) + 1024, "flops": case["count"] * 128 * (case["body"] + 3)}


def tolerance(case):
    """Against the same expression in 64 bits the float32 rows show a relative error of 6e-8 (largest 7e-7: rsqrt and exp after sums in another order);
    half-precision results show one rounding of the type, in 1e-5 of the values, where the float32 value before it lies next to a tie (5e-6 and 1.4e-5
    over all). Stated: four times that. The other programs are sums, products and comparisons in a given order."""
    kind = case["kind"]
    if kind == "head_rmsnorm" or case.get("dtype") == "bf16":
        return {"rel": 6e-5, "max": 1.6e-2}
    if case.get("dtype") == "f16":
        return {"rel": 2e-5, "max": 2e-3}
    if kind in ("add", "bmm4x4", "inv4x4", "candidates"):
        return "exact"
    return {"rel": 2.5e-7, "max": 3e-6}
