"""The streaming kernels' programs: finding the tile loops again (CPU: unrolling the stream must give back the program) and the kernels
themselves (GPU: the same bits as the tile kernels, which the other tests hold against the oracle)."""
import ctypes
import os
import sys

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import cases as C  # noqa: E402  (tests/cases.py)
from conftest import bits_equal, mismatch_report  # noqa: E402
from gint_b200 import bytecode, get_executor  # noqa: E402
from gint_b200 import opcodes as O  # noqa: E402
from gint_b200.host import capi, frontend as F  # noqa: E402
from gint_b200.host.utils import fill_tensor_info  # noqa: E402
from gint_b200.programs import load_records, recorded  # noqa: E402
from test_launch_route import EARLY, FLAT, WIDE as STREAMING, WIDE_VECTOR as STREAMING_VECTOR  # noqa: E402
from test_predecode_transforms import fold_repeated_loads, normalised  # noqa: E402

LOOP_BEGIN, REMAP, _, _, ACC_ADD, ACC_FMA, ACC_FMA_SQUARE, SQUARE, MUL_KEEP, SILU, LOOP_END = range(106, 117)
WIDE = 128
MINUS_ZERO = 0x80000000
TILES = {O.LoadGlobal1DF32: 128, O.StoreGlobal1DF32: 128, O.LoadGlobal1DF16: 128, O.StoreGlobal1DF16: 128, O.LoadGlobal1DBF16: 128,
         O.StoreGlobal1DBF16: 128, O.LoadGlobal1DU8: 128, O.LoadGlobal2DTF32: 32, O.StoreGlobal2DTF32: 32, O.LoadGlobal2DTF16: 32,
         O.StoreGlobal2DTF16: 32, O.LoadGlobal2DTBF16: 32, O.StoreGlobal2DTBF16: 32, O.LoadGlobal2DTU8: 32}


def stream(code, infos):
    """The stream with loops as (opcode, operand) pairs, or None."""
    code = np.ascontiguousarray(np.asarray(code, dtype=np.int32).reshape(-1))
    ti = capi.HTensorInfo()
    fill_tensor_info(ti, infos)
    n_max = code.size + 16
    ops, operands = (ctypes.c_int32 * n_max)(), (ctypes.c_uint32 * n_max)()
    n = capi.load_library().gint_debug_transform(code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), code.size, ctypes.byref(ti), len(infos),
                                                 8, 1, ops, operands, n_max)
    assert n >= 0, n
    return list(zip(ops[:n], operands[:n])) or None


def unroll(prog, flat_tiles=1):
    """Loops written out, forms undone. A sum that starts from -0 loses that start: its first AccAdd disappears with it."""
    out, i = [], 0
    while i < len(prog):
        op, operand = prog[i]
        if op == REMAP:
            i += 1
            continue
        if op != LOOP_BEGIN:
            out.append((op, operand))
            i += 1
            continue
        end = next(j for j in range(i, len(prog)) if prog[j][0] == LOOP_END)
        from_minus_zero = out and out[-1] == (O.LoadImm, MINUS_ZERO)
        if from_minus_zero:
            out.pop()
        for t in range(operand or flat_tiles):
            for op, arg in prog[i + 1:end]:
                if op >= WIDE:
                    op -= WIDE
                    out.append((op, arg + (t * TILES[op] << 4) if op in TILES else arg))
                elif op == ACC_ADD:
                    out.extend([] if from_minus_zero and t == 0 else [(O.FAdd, 0)])
                else:
                    out.extend({ACC_FMA: [(O.FMA, 0)], ACC_FMA_SQUARE: [(O.Dup, 0), (O.FMA, 0)], SQUARE: [(O.Dup, 0), (O.FMul, 0)],
                                MUL_KEEP: [("keep", 0)], SILU: [(O.Dup, 0), (O.FNeg, 0), (O.FExp, 0), (O.FAddImm, arg), (O.FRDiv, 0)]}[op])
        i = end + 1
    return out


def plain(code):
    """The program with Dup, <load>, (Swap), FMul written as the streaming form writes it: <load>, keep."""
    p, out, i = [(op, arg if op in TILES or op in (O.LoadImm, O.FAddImm, O.FMulImm, O.FMAImm, O.FPermW, O.FShuf2, O.DupBroadcastW, O.LoadImm4F, O.LoadImm4I,
                                                    O.FApprox) else 0) for op, arg in fold_repeated_loads(normalised(code))], [], 0
    while i < len(p):
        ops = [q[0] for q in p[i:i + 4]]
        if ops[:1] == [O.Dup] and len(ops) > 2 and ops[1] in TILES and "Store" not in O_NAME[ops[1]] and (ops[2] == O.FMul or ops[2:4] == [O.Swap, O.FMul]):
            out += [p[i + 1], ("keep", 0)]
            i += 3 if ops[2] == O.FMul else 4
        else:
            out.append(p[i])
            i += 1
    return out


O_NAME = {v: k for k, v in vars(O).items() if isinstance(v, int)}


def clean(prog):
    return [(op, arg if op in TILES or op in (O.LoadImm, O.FAddImm, O.FMulImm, O.FMAImm, O.FPermW, O.FShuf2, O.DupBroadcastW, O.LoadImm4F, O.LoadImm4I,
                                               O.FApprox) else 0) for op, arg in prog]


def test_unrolled_streams_are_the_recorded_programs():
    seen = 0
    for name in load_records():
        if name == "execute_everything":
            continue
        rec = recorded(name)
        s = stream(rec.bytecode, rec.tensor_infos)
        if s is None:
            continue
        seen += 1
        want = plain(rec.bytecode)
        loads = [op for op, _ in want if op in TILES]
        body = [op - WIDE for op, _ in s if op >= WIDE and op - WIDE in TILES]
        got = clean(unroll(s, len(loads) // max(1, len(body)) if s[0] == (LOOP_BEGIN, 0) else 1))
        assert got == want, name
    assert seen >= 5


@bytecode
def running_sum_times(x, s, out, REGW, WARP, n=1024, step=128, off2=0, body="add"):
    xb = F.make_block_1d(x, n, 1, 1, n, [n], [x.shape[0]])
    ob = F.make_block_1d(out, n, 1, 1, n, [n], [x.shape[0]])
    F.fpush(0.0)
    for off in range(0, n, step):
        F.fldg_1d(off, xb)
        if body == "read":        # the running value is read in the body: no loop
            F.fadd()
            F.dup()
            F.fstg_1d(off, ob)
        elif body == "shifted":   # the second access of a stored slot lies elsewhere
            F.fstg_1d(off, ob)
            F.fldg_1d(off + 256, ob)
            F.fadd()
        else:
            F.fadd()
    F.pop()
    F.halt()


@pytest.mark.parametrize("kw", [{"body": "read"}, {"body": "shifted"}, {"step": 256}])
def test_what_is_no_loop_has_no_stream(kw):
    t = C.to_interfaces([torch.zeros(4, 1024)] * 3)
    pd = running_sum_times.get_program(*t, **kw)
    assert stream(pd.program, pd.input_infos) is None


# ---------------------------------------------------------------------------------------------- on the GPU

@pytest.fixture(autouse=True)
def interpreter(request):
    """Many of these programs have a form, whose kernel would run them (tests/test_forms.py): off here."""
    if "gpu" not in request.keywords:
        yield
        return
    get_executor().set_option("forms", 0)
    yield
    get_executor().set_option("forms", 1)


def route_of(program, tensors, first, count, gathered=(), **kw):
    """The kernels that a launch of `program` on these tensors runs on (gint_debug_route)."""
    args = C.to_interfaces(tensors)
    pd = program.get_program(*args, **kw)
    code = np.ascontiguousarray(np.asarray(pd.program, dtype=np.int32).reshape(-1))
    ti = capi.HTensorInfo()
    fill_tensor_info(ti, pd.input_infos)
    order = list(getattr(pd, "input_indices", None) or range(len(pd.input_infos)))
    bases = (ctypes.c_uint64 * 8)(*[tensors[i].data_ptr() for i in order])
    mask = sum(1 << k for k, i in enumerate(order) if i in gathered)
    extent = max([tensors[i].numel() * tensors[i].element_size() for i in gathered], default=0)
    return capi.load_library().gint_debug_route(code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), code.size, ctypes.byref(ti), len(order), bases,
                                                first, count, mask, extent)


def both(launch):
    """What `launch` returns on the kernels of its route and on the tile kernels."""
    ex, got = get_executor(), []
    for on in (1, 0):
        ex.set_option("streaming", on)
        try:
            got.append([t.cpu() for t in launch()])
        finally:
            ex.set_option("streaming", 1)
    return got


def same_bits(launch):
    for a, b in zip(*both(launch)):
        assert bits_equal(a, b), mismatch_report(a, b)


def _perf_cases():
    import importlib.util
    spec = importlib.util.spec_from_file_location("timed_cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


EDGES = ([{"kind": "add", "n": n} for n in (1, 127, 128, 1024, 1025, 4096, 40003, 1048576 + 77)] +
         [{"kind": "gated_silu", "n": n, "dtype": d} for d in ("f32", "f16", "bf16") for n in (5, 512, 4000, 4097, 300001)] +
         [{"kind": "rmsnorm", "rows": r, "n": n} for r, n in ((3, 257), (5, 384), (1, 1024), (700, 1025), (33, 2029), (64, 4096), (2, 6000))] +
         [{"kind": "head_rmsnorm", "batch": b, "tokens": t, "heads": h, "dim": d} for b, t, h, d in ((1, 13, 1, 64), (2, 12, 3, 80), (1, 31, 2, 96), (2, 64, 5, 128))] +
         [{"kind": k, "rows": r, "n": n} for k in ("graph_gathered", "graph_plan") for r, n in ((10, 256), (77, 1024), (40, 1300), (9, 4095))])


@pytest.mark.gpu
@pytest.mark.parametrize("case", EDGES, ids=lambda c: "-".join(str(v) for v in c.values()))
def test_streaming_kernels_give_the_bits_of_the_tile_kernels(case):
    """(Flat programs of these sizes, and aligned rows of whole tiles, have the tile kernels as their route.)"""
    m = _perf_cases()

    def launch():
        r = m.run(m.prepare(dict(case, name="edge"), 7))
        return r if isinstance(r, tuple) else (r,)
    if case["kind"] == "head_rmsnorm" and case["dim"] == 128:   # the squares are added in another order; one bf16 rounding after it
        t = m.inputs(dict(case, name="edge"), 7)
        x = t["x"].double()
        want = (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * t["w"].double()).cpu()
        for (y,) in both(launch):
            torch.testing.assert_close(y.double(), want, rtol=2.0 ** -8 + 2.0 ** -18, atol=0.0)
    else:
        same_bits(launch)


@bytecode
def rmsnorm_f16(x, w, out, REGW, WARP):
    rows, n = x.shape
    tile = REGW * WARP
    xb, wb, ob = [F.make_block_1d(t, n, 1, 1, n, [n if t.ndim == 2 else 0], [rows]) for t in (x, w, out)]
    for off in range(0, n, tile):
        F.fldg_1d_f16(off, xb)
        F.dup()
        F.fmul()
        if off:
            F.fadd()
    F.warp_allreduce_fsum()
    F.dup()
    F.fperm_w(2, 3, 0, 1)
    F.fadd()
    F.dup()
    F.fperm_w(1, 0, 3, 2)
    F.fadd()
    F.fmulimm(1.0 / n)
    F.frsqrt()
    for off in range(0, n, tile):
        F.dup()
        F.fldg_1d_f16(off, xb)
        F.fmul()
        F.fldg_1d_f16(off, wb)
        F.fmul()
        F.fstg_1d_f16(off, ob)
    F.halt()


@pytest.mark.gpu
@pytest.mark.parametrize("rows,n,shift", [(3, 256, 0), (700, 1024, 0), (37, 1028, 0), (37, 1029, 0), (20, 4096, 0), (20, 4096, 1)])
def test_rows_of_half_precision(rows, n, shift):
    """Vector layout with a rearranged running sum (aligned rows) and natural layout (odd lengths, a base pointer off by one element):
    the bits of the tile kernels."""
    ex = get_executor()
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows * n + shift, device="cuda", generator=g).half()[shift:].view(rows, n)
    w = torch.rand(n, device="cuda", generator=g).half()
    got = []
    for on in (1, 0):
        ex.set_option("streaming", on)
        try:
            out = torch.zeros(rows, n, dtype=torch.float16, device="cuda")
            rmsnorm_f16(x, w, out, grid_dim=rows)
            got.append(out.cpu())
        finally:
            ex.set_option("streaming", 1)
    assert bits_equal(*got), mismatch_report(*got)
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True)) * w.double()
    torch.testing.assert_close(got[0].double(), want.cpu(), rtol=2e-3, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("first,count", [(0, 3), (5, 1), (2, 9)])
def test_streaming_range_and_in_place(first, count):
    """A range of the logical programs touches exactly its tiles (row programs on the streaming kernels, a flat program too small for
    them), and an output that overlaps an input, which keeps the tile kernels, gives the bits of the program as written."""
    from gint_b200.host.executor import _convert_arg
    m, ex = _perf_cases(), get_executor()
    g = torch.Generator(device="cuda").manual_seed(3)
    a, b = torch.randn(1500, device="cuda", generator=g), torch.randn(1500, device="cuda", generator=g)
    x, w = torch.randn(12, 700, device="cuda", generator=g), torch.randn(700, device="cuda", generator=g)
    got = []
    for on in (1, 0):
        ex.set_option("streaming", on)
        try:
            o1, o2 = torch.full((1500,), 9.0, device="cuda"), torch.full((12, 700), 9.0, device="cuda")
            ex.execute_range(m.add, [_convert_arg(t) for t in (o1, a, b)], first, count)
            ex.execute_range(m.rmsnorm, [_convert_arg(t) for t in (x, w, o2)], first, count)
            y = x.clone()
            m.rmsnorm(y, w, y, grid_dim=12)
            got.append([t.cpu() for t in (o1, o2, y)])
        finally:
            ex.set_option("streaming", 1)
    for p, q in zip(*got):
        assert bits_equal(p, q), mismatch_report(p, q)


N_FLAT = 2 ** 22 + 128 * 3000      # above the sizes from which flat programs run on the streaming kernels


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype", [("add", "f32"), ("gated_silu", "f16"), ("gated_silu", "bf16")])
@pytest.mark.parametrize("rest,shift", [(127, 0), (1, 0), (77, 0), (1024 + 640 + 3, 0), (77, 1), (130, (0, 1, 0))])
def test_flat_streaming(kind, dtype, rest, shift):
    """Flat launches: lengths that fill no last group of tiles, base pointers off by one element (the natural layout), and ranges that
    start and end inside the grid, which touch exactly their own elements. The bits of the tile kernels, guard bands included."""
    m, ex = _perf_cases(), get_executor()
    dt = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[dtype]
    n, shifts = N_FLAT + rest, shift if isinstance(shift, tuple) else (shift,) * 3
    g = torch.Generator(device="cuda").manual_seed(rest)
    a, b = [torch.randn(n + 64, device="cuda", generator=g).to(dt)[s:s + n] for s in shifts[1:]]
    program, kw, per = (m.add, {}, 128) if kind == "add" else (m.gated_silu, {"dtype": dtype}, 512)
    total = -(-n // per)
    aligned = not any(shifts)
    for first, count in ((0, total), (0, total - 3), (total - -(-32769 * 128 // per), -(-32769 * 128 // per)), (5, total - 9)):
        def launch():
            buffer = torch.full((n + 128,), 9.0, dtype=dt, device="cuda")
            out = buffer[64 + shifts[0]:64 + shifts[0] + n]
            assert route_of(program, [out, a, b], first, count, **kw) == (STREAMING_VECTOR if aligned else STREAMING) | FLAT
            ex.execute_range(program, C.to_interfaces([out, a, b]), first, count, cuda_stream=torch.cuda.current_stream().cuda_stream, **kw)
            return [buffer]
        same_bits(launch)


@bytecode
def rows_2dt(x, y, w, REGW, WARP, load="fldg_2dt", weight="fldg_2dt", store="fstg_2dt"):
    """rmsnorm of (rows, dim), four rows per logical program, one per width value."""
    T, H = x.shape
    xb, yb = [F.make_block_2d(t, [H, T], [1, t.strides[0]], [1, -(-T // REGW)], [0, REGW]) for t in (x, y)]
    wb = F.make_block_2d(w, [H, T], [1, 0], [1, -(-T // REGW)], [0, REGW])
    F.fpush(0.0)
    for c in range(0, H, WARP):
        getattr(F, load)(c, xb)
        F.dup()
        F.fma()
    F.warp_allreduce_fsum()
    F.fmulimm(1 / H)      # (one f32 each: the two immediates of FMAImm share a word)
    F.faddimm(1e-5)
    F.frsqrt()
    for c in range(0, H, WARP):
        F.dup()
        getattr(F, load)(c, xb)
        F.fmul()
        getattr(F, weight)(c, wb)
        F.fmul()
        getattr(F, store)(c, yb)
    F.halt()


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 37, 4000])
@pytest.mark.parametrize("dim", [64, 80, 128, 132, 192, 384, 396])
@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16", "u8"])
def test_streaming_2dt_rows(rows, dim, dtype):
    """Every element type of 2DT tiles. f32 and u8 sums, and sums over a number of tiles that is no multiple of four, have the bits of the
    tile kernels; the others, whose terms are added in another order, are held to a 64-bit reference within one rounding of the result's type."""
    dt = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "u8": torch.uint8}[dtype]
    suffix = {"f32": "", "u8": "_u8"}.get(dtype, "_" + dtype)
    g = torch.Generator(device="cuda").manual_seed(rows + dim)
    x = torch.randint(0, 256, (rows, dim), device="cuda", generator=g).to(dt) if dtype == "u8" else torch.randn(rows, dim, device="cuda", generator=g).to(dt)
    out_type = torch.float32 if dtype == "u8" else dt
    w = torch.rand(dim, device="cuda", generator=g).to(out_type)
    kw = {"load": "fldg_2dt" + suffix, "weight": "fldg_2dt" + ("" if dtype == "u8" else suffix), "store": "fstg_2dt" + ("" if dtype == "u8" else suffix)}

    def launch():
        y = torch.full((rows, dim), 9.0, dtype=out_type, device="cuda")
        r = route_of(rows_2dt, [x, y, w], 0, -(-rows // 4), **kw)
        tiles = -(-dim // 32)
        if dtype in ("f16", "bf16") and dim % 128 == 0:
            assert r == STREAMING_VECTOR
        else:
            assert (r == STREAMING) == (tiles >= {"f32": 6, "bf16": 6}.get(dtype, 10)) and r != STREAMING_VECTOR
        rows_2dt(x, y, w, grid_dim=-(-rows // 4), **kw)
        return [y]
    if dtype in ("f32", "u8") or -(-dim // 32) % 4 != 0:
        same_bits(launch)
        return
    xd = x.double()
    want = (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()).cpu()
    half_ulp = 2.0 ** (-8 if dtype == "bf16" else -11)      # relative; the f32 steps before it (sums of at most 384 terms, rsqrt) add below 2^-18
    for y, in both(launch):
        torch.testing.assert_close(y.double(), want, rtol=half_ulp + 2.0 ** -18, atol=2.0 ** -25 if dtype == "f16" else 0.0)   # (half of f16's smallest subnormal)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,rows,n,want", [("f16", 40, 2052, STREAMING_VECTOR), ("f16", 40, 2053, STREAMING), ("f16", 1, 2053, STREAMING), ("f32", 33, 2029, STREAMING), ("f32", 40, 1024, EARLY)])
def test_streaming_gathered_rows(dtype, rows, n, want):
    """Rows read through an index, on the kernels that their alignment allows: the bits of the rows gathered first."""
    m, ex = _perf_cases(), get_executor()
    dt, program = (torch.float16, rmsnorm_f16) if dtype == "f16" else (torch.float32, m.rmsnorm)
    g = torch.Generator(device="cuda").manual_seed(n)
    table, w = torch.randn(rows, n, device="cuda", generator=g).to(dt), torch.rand(n, device="cuda", generator=g).to(dt)
    idx = torch.randint(0, rows, (rows,), device="cuda", generator=g)
    copy = table[idx].contiguous()

    def launch(gather):
        out = torch.full((rows, n), 9.0, dtype=dt, device="cuda")
        if gather:
            assert route_of(program, [table, w, out], 0, rows, gathered=(0,)) == want
            ex.execute_gathered(program, C.to_interfaces([table, w, out]), rows, (0,), idx, cuda_stream=torch.cuda.current_stream().cuda_stream)
        else:
            program(copy, w, out, grid_dim=rows)
        return [out]
    same_bits(lambda: launch(True))
    (got,), (tile,) = both(lambda: launch(True))[0], both(lambda: launch(False))[1]
    assert bits_equal(got, tile), mismatch_report(got, tile)


@pytest.mark.gpu
def test_launch_info_reports_the_streaming_kernel():
    m, ex = _perf_cases(), get_executor()
    x, w, out = torch.zeros(100, 2029, device="cuda"), torch.zeros(2029, device="cuda"), torch.zeros(100, 2029, device="cuda")
    info = ex.launch_info(m.rmsnorm, [x, w, out], 100)
    assert (info["form"], info["streaming"], info["pool_size"], info["tiles_per_warp"], info["warps_per_block"]) == (0, 1, 3, 8, 1), info
    ex.set_option("streaming", 0)
    try:
        info = ex.launch_info(m.rmsnorm, [x, w, out], 100)
        assert info["streaming"] == 0 and info["pool_size"] == 4 and info["warps_per_block"] == 4, info
    finally:
        ex.set_option("streaming", 1)
