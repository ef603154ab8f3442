"""Form kernels: which programs and launches run on them (CPU, gint_debug_form) and that they give the interpreter's bits (GPU)."""
import ctypes
import random

import numpy as np
import pytest
import torch

import cases as C  # tests/cases.py
from conftest import bits_equal, mismatch_report
from gint_b200 import bytecode, get_executor
from gint_b200 import opcodes as O
from gint_b200.host import capi, frontend as F
from gint_b200.host.utils import fill_tensor_info
from test_streaming import _perf_cases

ROWS, LANES, HEADS, FLAT = 1, 2, 3, 4


def form(pd, bases, first=0, count=1, gather_mask=0, extent=1 << 30, logical=0, row=0, infos=None):
    """(form, warps per logical program, element offsets of `logical` by tensor slot)"""
    code = np.ascontiguousarray(np.asarray(pd.program, dtype=np.int32).reshape(-1))
    ti = capi.HTensorInfo()
    fill_tensor_info(ti, pd.input_infos)
    n = len(pd.input_infos)
    if infos:
        infos(ti)
    off = (ctypes.c_uint32 * 8)()
    r = capi.load_library().gint_debug_form(code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), code.size, ctypes.byref(ti), n, (ctypes.c_uint64 * 8)(*bases),
                                            first, count, gather_mask, extent, logical, row, off)
    assert r >= 0, r
    return r & 255, r >> 8, list(off[:n]), ti


@bytecode
def rows_program(x, w, r, z, REGW, WARP, n=1024, tiles=None, reduce="squares", steps="mean", scale=True, silu=False, c=1.0, add=False, first="load"):
    """The shapes that a row program can have: z = [silu](s * x [* w]) [+ r] with s from a sum over x; without `scale` z = s."""
    rows = x.shape[0]
    xb, wb, rb = [F.make_block_1d(t, n, 1, 1, n, [t.strides[0] if t.ndim == 2 else 0], [rows]) for t in (x, w, r)]
    zb = F.make_block_1d(z, n if scale else 1, 1, 1, n if scale else 1, [z.strides[0]], [rows])
    offs = range(0, 128 * (tiles or -(-n // 128)), 128)
    if reduce == "fma" or first == "zero":
        F.fpush(0.0)
    for off in offs:
        F.fldg_1d(off, xb)
        if reduce == "squares":
            F.dup()
            F.fmul()
        if reduce == "fma":
            F.dup()
            F.fma()
        elif off or first == "zero":
            F.fadd()
    if steps != "none":
        F.warp_allreduce_fsum()
        F.dup()
        F.fperm_w(2, 3, 0, 1)
        F.fadd()
        F.dup()
        F.fperm_w(1, 0, 3, 2)
        F.fadd()
    if steps == "mean":
        F.fmulimm(1.0 / n)
        F.faddimm(1e-6)
        F.frsqrt()
    elif steps == "others":
        F.dup()
        F.fperm_w(0, 0, 3, 1)
        F.fadd()
        F.fmaimm(0.25, 1.5)
        F.fneg()
        F.fmulimm(-0.5)
        F.fsqrt()
        F.frcp()
    if not scale:
        F.fstg_1d(0, zb)
        F.halt()
        return
    for off in offs:
        F.dup()
        F.fldg_1d(off, xb)
        F.fmul()
        if w is not r:
            F.fldg_1d(off, wb)
            F.fmul()
        if silu:
            F.dup()
            F.fneg()
            F.fexp()
            F.faddimm(c)
            F.frdiv()
        if add:
            F.fldg_1d(off, rb)
            F.fadd()
        F.fstg_1d(off, zb)
    F.pop()
    F.halt()


FAR = [(t + 1) << 36 for t in range(8)]


def program(rows=64, n=1024, w_rows=False, **kw):
    t = C.to_interfaces([torch.empty(rows, n), torch.empty(rows, n) if w_rows else torch.empty(n), torch.empty(rows, n), torch.empty(rows, n)])
    return rows_program.get_program(*t, n=n, **kw)


@pytest.mark.parametrize("kw", [{}, {"silu": True}, {"add": True}, {"silu": True, "add": True}, {"reduce": "sum"}, {"reduce": "fma"}, {"first": "zero"}, {"steps": "others"},
                                {"steps": "none"}, {"scale": False}, {"n": 129}, {"n": 256}, {"n": 257}, {"w_rows": True}, {"tiles": 9}])
def test_row_programs_have_the_form(kw):
    assert form(program(**kw), FAR, count=64)[0] == ROWS


def test_what_a_launch_on_the_form_needs():
    pd = program()
    assert form(pd, FAR, count=64)[0] == ROWS
    assert form(pd, [FAR[0] + 4, FAR[1] + 12, FAR[2], FAR[3] + 8], count=64)[0] == ROWS          # any element may be the first
    assert form(pd, [FAR[0] + 2] + FAR[1:], count=64)[0] == 0                                     # ... but no part of one
    end = 4 * 64 * 1024
    for bases, want in ((FAR[:3] + [FAR[0]], 0), (FAR[:3] + [FAR[0] + end - 4], 0), (FAR[:3] + [FAR[0] + end], ROWS), (FAR[:3] + [FAR[1] + 4092], 0)):
        assert form(pd, bases, count=64)[0] == want                                               # what is stored is read by no other logical program
    assert form(pd, FAR, first=(1 << 31) - 60, count=64)[0] == 0                                  # logical programs are counted in 31 bits
    assert form(program(n=20000), FAR, count=64)[0] == 0                                          # two rows and the weights in shared memory
    assert form(program(rows=100000, n=300, scale=False), FAR, count=100000)[0] == ROWS           # sums, however short and many
    assert form(program(n=8192, silu=True, add=True), FAR, count=296)[0] == ROWS                  # one team per SM
    assert form(program(n=8192, silu=True, add=True), FAR, count=297)[0] == 0


@pytest.mark.parametrize("n,rows,kw,warps", [(384, 10, {}, 1), (385, 296, {}, 4), (385, 297, {}, 1), (996, 5000, {}, 1), (1000, 5000, {}, 4), (1001, 5000, {}, 1), (1399, 5000, {}, 1), (1401, 5000, {}, 4),
                                             (1000, 5000, {"steps": "others"}, 1), (1536, 5000, {"silu": True, "add": True}, 1), (1537, 5000, {"silu": True, "add": True}, 4),
                                             (1792, 5000, {"silu": True, "add": True}, 4), (2200, 5000, {"scale": False}, 1), (2600, 5000, {"scale": False}, 4)])
def test_warps_per_row(n, rows, kw, warps):
    assert form(program(rows=rows, n=n, **kw), FAR, count=rows)[:2] == (ROWS, warps)


def row_layout(pd, bases, count):
    """gint_debug_rows: the launch's numbers and, by operand, (elements read, byte offset of the row, staged once), or None"""
    code = np.ascontiguousarray(np.asarray(pd.program, dtype=np.int32).reshape(-1))
    ti = capi.HTensorInfo()
    fill_tensor_info(ti, pd.input_infos)
    out = (ctypes.c_uint32 * 17)()
    r = capi.load_library().gint_debug_rows(code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), code.size, ctypes.byref(ti), len(pd.input_infos), (ctypes.c_uint64 * 8)(*bases), count, out)
    assert r >= 0, r
    names = ("team", "teams", "depth", "tiles", "full", "stage", "stationary", "smem")
    return (dict(zip(names, out[:8])), [tuple(out[8 + 3 * s:11 + 3 * s]) for s in range(3)]) if r else None


def last_element_read(tiles, full, left, team, reduce):
    """The largest element of a staged row that the threads of a team read (rows_reduce, rows_map in gint_rows.cuh), where the row has `left` elements."""
    values = 4 // team
    U = {1: 8 if reduce else 4, 4: 2}[values]
    last = -1
    for at in {lane + 32 * values * warp for warp in range(team) for lane in (0, 31)}:
        k = 0
        while k < tiles:
            masked = k + U > full
            for u in range(U):
                for i in range(values):
                    e = at + 128 * (k + u) + 32 * i
                    if not masked or e < left:
                        last = max(last, e)
            k += U
    return last


@pytest.mark.parametrize("n,tiles,rows", [(12000, 65, 5000), (6001, 41, 5000), (20000, 137, 5000), (1500, 5, 5000), (1500, 5, 100), (700, 3, 9), (1024, 9, 64), (1029, None, 64), (4096, None, 700),
                                          (129, None, 9000), (9000, None, 3)])
@pytest.mark.parametrize("kw", [{}, {"scale": False}, {"silu": True, "add": True}, {"w_rows": True, "add": True}])
def test_staged_rows_hold_what_is_read(n, tiles, rows, kw):
    """Rows of which the program sums a part, the whole, or more than there is: no thread reads behind what was staged, and the stages lie in the block's memory."""
    layout = row_layout(program(rows=rows, n=n, tiles=tiles, **kw), FAR, rows)
    if layout is None:
        assert n > 4096 or (n < 256 and not kw.get("scale", True))      # (two tiles that are only summed are no loop)
        return
    a, operands = layout
    staged = min(n, 128 * a["tiles"])
    areas = {0: [], 1: []}
    for s, (left, area, once) in enumerate(operands):
        if left:
            for reduce in ((True, False) if s == 0 else (False,)):
                assert last_element_read(a["tiles"], a["full"], left, a["team"], reduce) < staged
            areas[once].append((area, area + (4 * staged + 12 + 15 & ~15)))      # (a row may start at any of the four elements of its first 16 bytes)
    for once, end in ((0, a["stage"] - 16), (1, a["stationary"])):
        for (_, e), (b, _) in zip(sorted(areas[once]), sorted(areas[once])[1:] + [(end, None)]):
            assert e <= b
    assert a["stationary"] + a["teams"] * (a["depth"] * (a["stage"] + 8) + (1024 if a["team"] > 1 else 0)) + 8 <= a["smem"] <= 227 * 1024


def test_a_program_too_long_for_the_tile_kernels_has_no_form():
    """What is refused must not depend on the route: the tile kernels keep the whole program in shared memory."""
    assert form(flat(n=128 * 5000, tiles=5000, op="fadd"), FAR, count=1)[0] == FLAT
    assert form(flat(n=128 * 12000, tiles=12000, op="fadd"), FAR, count=1)[0] == 0


def test_gathered_rows_of_a_form():
    """An index replaces the digit of the innermost batch dimension. Where that has one row, the index still moves the row."""
    pd = program()
    assert form(pd, FAR, count=64, gather_mask=1)[0] == ROWS
    assert form(pd, FAR, count=64, gather_mask=8)[0] == 0                                         # not what is stored
    assert form(program(rows=1), FAR, count=1, gather_mask=1)[0] == 0
    assert form(program(rows=1), FAR, count=1)[0] == ROWS
    assert form(pd, FAR, count=64, gather_mask=2)[0] == ROWS                                      # (weights: the same row for every index)


def decode(ti, t, r, gathered, row):
    """decode_tiles (gint_interp.cuh) for a slot whose block grid does not cut dimension 1"""
    off, step2 = 0, ti.block_grid_steps[t][1] * ti.block_shape_stride_2[t][1]
    if ti.block_grid_dims[t][1] != 1:
        off, r = off + r % ti.block_grid_dims[t][1] * step2, r // ti.block_grid_dims[t][1]
    for j in range(4):
        size, stride = ti.batch_shape[t][j], ti.batch_strides[t][j]
        b = r % size
        off += (row if gathered and j == 0 else b) * stride
        r //= size
    return off & 0xFFFFFFFF


@pytest.mark.parametrize("seed", range(12))
def test_offsets_are_those_of_the_descriptor_decode(seed):
    """Digits of any size and order, slots that do not move, leftover digits, a gathered digit."""
    pd = program()
    rng = random.Random(seed)
    gather = seed % 3 == 0
    sizes = [rng.choice([1, 1, 2, 3, 7, 64, 1000, 4099]) for _ in range(5)]      # grid dimension 2, four batch dimensions
    if gather:
        sizes[1] = rng.randint(2, 50)
    moving = [t for t in (0, 1, 3) if t != 1 or rng.random() < 0.5]
    strides = {t: [rng.randint(1, 40) if t in moving else 0 for _ in range(5)] for t in (0, 1, 3)}
    plain = rng.random() < 0.5                                                    # a slot that does not move may have any digits

    def infos(ti):
        for t in (0, 1, 3):                                                       # (slot 2 is not accessed by this program)
            one = plain and t not in moving
            ti.block_grid_dims[t][1] = 1 if one else sizes[0]
            ti.block_grid_steps[t][1], ti.block_shape_stride_2[t][1] = strides[t][0], 1
            for j in range(4):
                ti.batch_shape[t][j], ti.batch_strides[t][j] = (1 if one else sizes[j + 1]), strides[t][j + 1]
    total = min(int(np.prod(sizes, dtype=np.float64)) * 2, (1 << 31) - 2)
    for logical in [0, total // 2] + [rng.randrange(total) for _ in range(20)]:
        kind, _, off, ti = form(pd, FAR, first=logical, count=1, gather_mask=1 if gather else 0, logical=logical, row=13, infos=infos)
        reach = max(sum((s - 1) * d for s, d in zip(sizes, strides[t])) + 1024 for t in moving)
        assert (kind == ROWS) == (reach < (1 << 31) - 8192 and 4 * reach < 1 << 36), (sizes, strides)
        for t in (0, 1, 3) if kind else ():
            assert off[t] == decode(ti, t, logical, gather and t == 0, 13), (t, logical, sizes)


def matrix_program(kind, batch=1000, stride=16):
    m = _perf_cases()
    t = C.to_interfaces([torch.empty(batch, 16)] * (3 if kind == "bmm4x4" else 2))
    pd = getattr(m, kind).get_program(*t)
    for info in pd.input_infos:
        info.block_shape_stride_1[1] = stride
    return pd


@pytest.mark.parametrize("kind,n_slots", [("bmm4x4", 3), ("inv4x4", 2)])
def test_what_a_launch_of_a_lane_program_needs(kind, n_slots):
    pd, out = matrix_program(kind), n_slots - 1
    tiles, size = 32, 64 * 1000
    assert form(pd, FAR, count=tiles)[:2] == (LANES, 1)
    assert form(pd, FAR, first=30, count=2)[0] == LANES and form(pd, FAR, first=30, count=3)[0] == 0      # tiles behind the grid wrap
    assert form(matrix_program(kind, stride=20), FAR, count=tiles)[0] == LANES
    assert form(matrix_program(kind, stride=18), FAR, count=tiles)[0] == 0 and form(matrix_program(kind, stride=12), FAR, count=tiles)[0] == 0
    assert form(pd, FAR, count=tiles, gather_mask=1)[0] == 0
    for t in range(n_slots):
        assert form(pd, [b + (8 if k == t else 0) for k, b in enumerate(FAR)], count=tiles)[0] == 0       # 16-byte rows
        assert form(pd, [b + (16 if k == t else 0) for k, b in enumerate(FAR)], count=tiles)[0] == LANES
    for at, want in ((0, 0), (size - 16, 0), (size, LANES), (-size, LANES), (16 - size, 0)):
        assert form(pd, [FAR[0] + at if k == out else b for k, b in enumerate(FAR)], count=tiles)[0] == want
    if kind == "bmm4x4":
        assert form(pd, [FAR[0], FAR[0], FAR[2]], count=tiles)[0] == LANES                                # a @ a
    for info, change in ((0, ("block_shape_stride_2", [15, 1])), (1, ("block_shape_stride_2", [16, 2])), (0, ("block_grid_steps", [31, 0])), (out, ("elm_size", 2)),
                         (1, ("block_grid_dims", [31, 1]))):
        pd = matrix_program(kind)
        infos = [type(i)(**vars(i)) for i in pd.input_infos]
        setattr(infos[info], *change)
        pd.input_infos[:] = infos
        assert form(pd, FAR, count=tiles)[0] == 0, (info, change)


@pytest.mark.parametrize("kind", ["bmm4x4", "inv4x4"])
def test_a_lane_program_is_one_to_the_last_operand(kind):
    pd = matrix_program(kind)
    code = np.asarray(pd.program, dtype=np.int32).reshape(-1, 2)
    ops = {O.LoadGlobal2DWF32, O.StoreGlobal2DWF32, O.DupBroadcastW, O.FPermW, O.FShuf2, O.LoadImm4F}
    for i in range(len(code) - 1):
        changed = code.copy()
        if code[i, 0] in ops:
            changed[i, 1] ^= 1 if code[i, 0] in (O.DupBroadcastW, O.FPermW, O.FShuf2, O.LoadImm4F) else 64
        elif code[i, 0] in (O.FAdd, O.FMul, O.FSub, O.FRSub):
            changed[i, 0] = O.FDiv
        else:
            continue
        assert form(type(pd)(changed, pd.input_infos), FAR, count=32)[0] == 0, i


@bytecode
def heads_program(x, y, w, REGW, WARP, fused=True, load="fldg_2dt_bf16", reduce="fma"):
    """rmsnorm over the last dimension of (batch, heads, tokens, dim) views, four tokens per logical program."""
    B, NH, T, H = x.shape
    xb, yb = [F.make_block_2d(t, [H, T], [t.strides[-1], t.strides[-2]], [1, -(-T // REGW)], [0, REGW], [t.strides[0], t.strides[1]], [B, NH]) for t in (x, y)]
    wb = F.make_block_2d(w, [H, T], [w.strides[-1], 0], [1, -(-T // REGW)], [0, REGW], [0, 0], [B, NH])
    F.fpush(0.0)
    for c in range(0, H, WARP):
        getattr(F, load)(c, xb)
        F.dup()
        if reduce == "fma":
            F.fma()
        else:
            F.fmul()
            F.fadd()
    F.warp_allreduce_fsum()
    if fused:
        F.fmaimm(1 / H, 1e-5)
    else:
        F.fmulimm(1 / H)
        F.faddimm(1e-5)
    F.frsqrt()
    for c in range(0, H, WARP):
        F.dup()
        getattr(F, load)(c, xb)
        F.fmul()
        getattr(F, load)(c, wb)
        F.fmul()
        getattr(F, load.replace("fldg", "fstg"))(c, yb)
    F.halt()


def head_views(batch, tokens, heads, dim, device="cpu", dtype=torch.bfloat16):
    return [torch.empty(batch, tokens, heads, dim, dtype=dtype, device=device).transpose(1, 2) for _ in range(2)] + [torch.empty(dim, dtype=dtype, device=device)]


def head_program(*shape, **kw):
    return heads_program.get_program(*C.to_interfaces(head_views(*shape, dtype=kw.pop("dtype", torch.bfloat16))), **kw)


@pytest.mark.parametrize("dim,kw,want", [(64, {}, HEADS), (33, {}, HEADS), (80, {"fused": False}, HEADS), (128, {}, HEADS), (32, {}, 0), (129, {}, 0), (128, {"reduce": "square"}, 0),
                                         (128, {"load": "fldg_2dt_f16", "dtype": torch.float16}, 0)])
def test_head_programs_have_the_form(dim, kw, want):
    assert form(head_program(2, 37, 3, dim, **kw), FAR, count=60)[0] == want


def test_what_a_launch_of_heads_needs():
    pd, size = head_program(2, 37, 3, 64), 2 * 2 * 37 * 3 * 64
    assert form(pd, [FAR[0] + 2, FAR[1] + 6, FAR[2] + 2], count=60)[0] == HEADS
    assert form(pd, [FAR[0] + 1] + FAR[1:], count=60)[0] == 0
    assert form(pd, FAR, count=60, gather_mask=1)[0] == 0
    for at, want in ((0, 0), (size - 2, 0), (size, HEADS)):                       # (the last four rows of a head end with its tokens)
        assert form(pd, [FAR[0], FAR[0] + at, FAR[2]], count=60)[0] == want


@pytest.mark.parametrize("shape", [(2, 37, 3, 64), (1, 8, 5, 128), (3, 4, 1, 96), (1, 1, 1, 80)])
def test_a_whole_launch_of_heads_takes_every_logical_program_once(shape):
    """The offsets of a launch of the whole grid are those of its logical programs, in the order of the addresses; a part keeps their numbers."""
    pd = head_program(*shape)
    total = shape[0] * shape[2] * -(-shape[1] // 4)
    offsets = [form(pd, FAR, count=total, logical=r)[2] for r in range(total)]
    want = [[decode(form(pd, FAR, count=total)[3], t, r, False, 0) for t in range(3)] for r in range(total)]
    assert sorted(offsets) == sorted(want) and [o[0] for o in offsets] == sorted(w[0] for w in want)
    for r in range(0, total - 1, 3):
        assert form(pd, FAR, first=r, count=1, logical=r)[2] == want[r]


@bytecode
def flat_program(x, y, z, REGW, WARP, op="silu_fmul", dtype="f32", tiles=1, start=0, c=1.0):
    n, = x.shape
    suffix, block = "" if dtype == "f32" else "_" + dtype, 128 * tiles
    xb, yb, zb = [F.make_block_1d(t, t.shape[0], t.strides[0], -(-n // block), block) for t in (x, y, z)]
    for off in range(start, start + block, 128):
        getattr(F, "fldg_1d" + suffix)(off, xb)
        if op.startswith("silu"):
            F.dup()
            F.fneg()
            F.fexp()
            F.faddimm(c)
            F.frdiv()
        if op != "silu":
            getattr(F, "fldg_1d" + suffix)(off, yb)
            getattr(F, op.replace("silu_", ""))()
        getattr(F, "fstg_1d" + suffix)(off, zb)
    F.halt()


TYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def flat(n=5000, ny=None, stride=1, **kw):
    t = [torch.empty(k * stride, dtype=TYPES[kw.get("dtype", "f32")])[::stride] for k in (n, ny or n, n)]
    return flat_program.get_program(*C.to_interfaces(t), **kw)


@pytest.mark.parametrize("kw,want", [({}, FLAT), ({"op": "fadd"}, FLAT), ({"op": "fmul", "dtype": "f16"}, FLAT), ({"op": "silu", "dtype": "bf16"}, FLAT), ({"op": "silu_fadd", "tiles": 4}, FLAT),
                                     ({"op": "fsub"}, 0), ({"start": 128}, 0), ({"ny": 4999}, 0), ({"stride": 2}, 0), ({"n": 1}, FLAT)])
def test_flat_programs_have_the_form(kw, want):
    assert form(flat(**kw), FAR, count=1)[0] == want


def test_what_a_flat_launch_needs():
    pd, size = flat(), 4 * 5000
    for t in range(3):
        assert form(pd, [b + (4 if k == t else 0) for k, b in enumerate(FAR)], count=40)[0] == 0          # 16-byte groups
        assert form(pd, [b + (16 if k == t else 0) for k, b in enumerate(FAR)], count=40)[0] == FLAT
    assert form(pd, FAR, first=39, count=1)[0] == FLAT and form(pd, FAR, first=39, count=2)[0] == 0
    assert form(pd, FAR, count=40, gather_mask=1)[0] == 0
    for at, want in ((0, FLAT), (16, 0), (size - 16, 0), (size, FLAT)):                                   # in place, but not shifted
        assert form(pd, [FAR[0], FAR[1], FAR[0] + at], count=40)[0] == want


# ---------------------------------------------------------------------------------------------- on the GPU

def both(launch):
    ex, got = get_executor(), []
    for on in (1, 0):
        ex.set_option("forms", on)
        try:
            got.append([t.cpu() for t in launch()])
        finally:
            ex.set_option("forms", 1)
    return got


def same_bits(launch):
    for a, b in zip(*both(launch)):
        assert bits_equal(a, b), mismatch_report(a, b)


def runs_on_form(program_, tensors, rows, **kw):
    return get_executor().launch_info(program_, C.to_interfaces(tensors), rows, **kw)["form"] == ROWS


@pytest.mark.gpu
def test_launch_info_describes_the_launch_of_a_form():
    """Blocks, threads and shared memory of the launch itself, and none of them without the form."""
    ex, m = get_executor(), _perf_cases()
    x, w, out = torch.zeros(16384, 4096, device="cuda"), torch.zeros(4096, device="cuda"), torch.zeros(16384, 4096, device="cuda")
    t = C.to_interfaces([x, w, out])
    a, _ = row_layout(m.rmsnorm.get_program(*t), FAR, 16384)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    info = ex.launch_info(m.rmsnorm, t, 16384)
    assert (info["form"], info["form_grid_blocks"], info["form_threads"], info["form_smem_bytes"]) == (ROWS, sms, 32 * a["team"] * a["teams"], a["smem"])
    ex.set_option("forms", 0)
    try:
        info = ex.launch_info(m.rmsnorm, t, 16384)
    finally:
        ex.set_option("forms", 1)
    assert (info["form"], info["form_grid_blocks"], info["form_threads"], info["form_smem_bytes"]) == (0, 0, 0, 0)
    n = 40003
    x, y, z = [torch.zeros(n, device="cuda") for _ in range(3)]
    info = ex.launch_info(flat_program, C.to_interfaces([x, y, z]), -(-n // 128), op="fadd")
    assert (info["form"], info["form_grid_blocks"], info["form_threads"], info["form_smem_bytes"]) == (FLAT, -(-(n // 4) // 256), 256, 0)


KEPT = []
SHAPES = [(1, 129), (3, 255), (700, 256), (5, 257), (40, 384), (7, 513), (300, 1000), (33, 1024), (2000, 1025), (9, 2029), (400, 2304), (20, 4095), (150, 4096), (5, 6001), (3, 9000)]
ALIGNED = [(1, 132), (700, 256), (40, 384), (300, 1000), (2000, 1024), (9, 2028), (400, 2304), (150, 4096), (5000, 644), (3, 9000)]   # four elements at a time


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [{}, {"silu": True, "add": True}, {"silu": True, "c": 0.5}, {"add": True, "reduce": "fma"}, {"reduce": "sum", "steps": "others"}, {"scale": False}, {"reduce": "sum", "steps": "total", "scale": False},
                                {"scale": False, "reduce": "sum", "first": "zero"}, {"steps": "none"}], ids=str)
def test_rows_give_the_bits_of_the_interpreter(kw):
    """Row lengths around whole tiles and groups of tiles, one and four warps per row, rows and base pointers at any element."""
    for k, (rows, n) in enumerate(SHAPES + ALIGNED):
        g = torch.Generator(device="cuda").manual_seed(k)
        pad = [k % 4, (k // 2) % 4, (k + 1) % 4, (k + 2) % 3] if k < len(SHAPES) else [4, 0, 8, 3]
        x, w, r, z = [torch.randn(rows * n + 8, device="cuda", generator=g)[p:p + rows * n].view(rows, n) for p in pad]
        w = w[0]

        def launch():
            out = torch.full((rows * n + 8,), 9.0, device="cuda")
            o = out[pad[3] + 1:pad[3] + 1 + rows * n].view(rows, n)
            rows_program(x, w, r, o, grid_dim=rows, n=n, **kw)
            return [out]
        assert runs_on_form(rows_program, [x, w, r, z], rows, n=n, **kw) == (n > 256 or kw.get("scale", True)), (rows, n)   # (two tiles that are only summed are no loop)
        same_bits(launch)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,n,tiles", [(9, 700, 3), (100, 1500, 5), (2000, 1500, 5), (2000, 1536, 7), (2000, 6001, 41), (400, 12000, 65), (1000, 8192, 33), (64, 1024, 9)])
@pytest.mark.parametrize("kw", [{}, {"scale": False}, {"silu": True, "add": True}, {"reduce": "fma", "add": True}], ids=str)
def test_rows_of_which_a_part_is_summed(rows, n, tiles, kw):
    """Programs over a part of their rows, whose number of tiles is no multiple of a group; what lies behind is left alone."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x, r = torch.randn(rows, n, device="cuda", generator=g), torch.randn(rows, n, device="cuda", generator=g)
    x[:, 128 * tiles:] = float("nan")

    def launch():
        out = torch.full((rows, n), 9.0, device="cuda")
        rows_program(x, r[0], r, out, grid_dim=rows, n=n, tiles=tiles, **kw)
        return [out]
    assert runs_on_form(rows_program, [x, r[0], r, x], rows, n=n, tiles=tiles, **kw) == (n < 12000 or not kw.get("silu"))      # (one team per SM)
    same_bits(launch)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1028, 1030])
def test_rows_with_extreme_values(n):
    """Single elements and (1028) four at a time. SiLU's quotient where its plain steps do not hold: zeros of both signs, subnormal and huge values, infinities, NaN, every size of exp(-x)."""
    rows = 64
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(rows, n, device="cuda", generator=g) * torch.logspace(-40, 38, rows, device="cuda")[:, None]
    x[:, 5], x[:, 6], x[::3, 7], x[::5, 8], x[::7, 9] = 0.0, -0.0, float("inf"), float("-inf"), float("nan")
    w = torch.randn(n, device="cuda", generator=g) * torch.logspace(-30, 3, n, device="cuda")
    for kw in ({"steps": "none", "reduce": "sum", "silu": True}, {"silu": True, "add": True}, {"reduce": "fma"}, {}):
        def launch():
            z = torch.empty(rows, n, device="cuda")
            rows_program(x, w, x, z, grid_dim=rows, n=n, **kw)
            return [z]
        same_bits(launch)


@pytest.mark.gpu
def test_silu_of_any_bits():
    """A million random bit patterns and a million ordinary values: 8 * w through SiLU (x = 1 everywhere, eight tiles, no steps)."""
    rows, n = 1024, 1024
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.ones(rows, n, device="cuda")
    for w in (torch.randint(-2 ** 31, 2 ** 31, (rows, n), device="cuda", generator=g).to(torch.int32).view(torch.float32), torch.randn(rows, n, device="cuda", generator=g)):
        def launch():
            z = torch.empty(rows, n, device="cuda")
            rows_program(x, w, x, z, grid_dim=rows, n=n, steps="none", reduce="sum", silu=True)
            return [z]
        same_bits(launch)


@pytest.mark.gpu
def test_silu_of_all_bits():
    """Every 32-bit value through SiLU, in the order of the bits, so that most groups take the plain steps together."""
    ex, n = get_executor(), 1 << 26
    st, z = torch.cuda.current_stream().cuda_stream, torch.empty(2, n, device="cuda")
    for k in range(64):
        x = torch.arange(k * n - (1 << 31), (k + 1) * n - (1 << 31), dtype=torch.int64, device="cuda").to(torch.int32).view(torch.float32)
        for on in (1, 0):
            ex.set_option("forms", on)
            try:
                flat_program(x, x, z[on], grid_dim=n // 128, op="silu", cuda_stream=st)
            finally:
                ex.set_option("forms", 1)
        assert torch.equal(z[0].view(torch.int32), z[1].view(torch.int32)), k


@pytest.mark.gpu
@pytest.mark.parametrize("c", [-1.0, -0.0])
def test_silu_where_the_divisor_is_zero(c):
    """x / (exp(-x) + c): a sum that cancels, or that both terms leave at zero, is +0, and the sign of the quotient is that of x."""
    n = 1024
    v = torch.tensor([1e-10, -1e-10, 1e-30, -1e-42, 0.0, -0.0, 3e-8, -3e-8, 150.0, 1e30, float("inf"), -150.0, float("-inf"), float("nan"), 1.0, -1.0], device="cuda")
    v = torch.cat([v, v.roll(3), v.repeat_interleave(4)]).repeat(11)[:n].contiguous()
    x = torch.ones(4, n, device="cuda")

    def launch():
        z, y = torch.empty(4, n, device="cuda"), torch.empty(n, device="cuda")
        rows_program(x, v / 8, x, z, grid_dim=4, n=n, steps="none", reduce="sum", silu=True, c=c)
        flat_program(v, v, y, grid_dim=n // 128, op="silu", c=c)
        return [z, y]
    assert runs_on_form(rows_program, [x, v, x, x], 4, n=n, steps="none", reduce="sum", silu=True, c=c)
    assert get_executor().launch_info(flat_program, C.to_interfaces([v, v, v.clone()]), n // 128, op="silu", c=c)["form"] == FLAT
    same_bits(launch)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,n", [(40, 1025), (400, 384), (30, 4096)])
def test_gathered_and_partial_launches_of_rows(rows, n):
    m, ex = _perf_cases(), get_executor()
    g = torch.Generator(device="cuda").manual_seed(n)
    table, x, w = torch.randn(rows + 5, n, device="cuda", generator=g)[:rows], torch.randn(rows, n, device="cuda", generator=g), torch.randn(n, device="cuda", generator=g)
    idx = torch.randint(-rows, rows, (rows,), device="cuda", generator=g)
    idx[0], idx[1], idx[2] = rows + 100, -rows - 7, -1        # clamped, clamped, from the end
    st = torch.cuda.current_stream().cuda_stream

    def gathered():
        z = torch.full((rows, n), 9.0, device="cuda")
        ex.execute_gathered(m.rmsnorm_silu_residual, C.to_interfaces([z, x, w, table]), rows, (3,), idx, cuda_stream=st)
        return [z]
    same_bits(gathered)

    def part():
        z = torch.full((rows, n), 9.0, device="cuda")
        ex.execute_range(m.rmsnorm, C.to_interfaces([x, w, z]), 3, rows - 7, cuda_stream=st)
        y = x.clone()
        m.rmsnorm(y, w, y, grid_dim=rows)                      # in place: the interpreter
        return [z, y]
    same_bits(part)


@pytest.mark.gpu
def test_rows_in_a_graph_and_on_few_blocks():
    m, ex = _perf_cases(), get_executor()
    x, w, z = torch.randn(500, 777, device="cuda"), torch.randn(777, device="cuda"), torch.zeros(500, 777, device="cuda")
    m.rmsnorm(x, w, z, grid_dim=500)
    want = z.clone()
    graph = torch.cuda.CUDAGraph()
    KEPT.append(graph)      # (torch allocates its capture state with the first graph alive and frees it with the last: other tests count allocations)
    with torch.cuda.graph(graph):
        m.rmsnorm(x, w, z, grid_dim=500, cuda_stream=torch.cuda.current_stream().cuda_stream)
    z.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert bits_equal(z.cpu(), want.cpu())
    ex.set_option("max_blocks", 3)
    try:
        z.zero_()
        m.rmsnorm(x, w, z, grid_dim=500)
        assert bits_equal(z.cpu(), want.cpu())
    finally:
        ex.set_option("max_blocks", 0)
    assert ex.device_status()["code"] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows,n", [(700, 4096), (20000, 4096), (5000, 256), (300000, 256)])
def test_a_wait_that_runs_out_is_reported(rows, n):
    """Four warps per row and one: with no time to wait, teams give up while their first rows are on the way. The launch ends, no row is
    written, and every launch after it fails until the status is read, which says why."""
    ex = get_executor()
    x, w = torch.randn(rows, n, device="cuda"), torch.randn(n, device="cuda")
    z, want = torch.full((rows, n), 9.0, device="cuda"), torch.empty(rows, n, device="cuda")
    rows_program(x, w, x, want, grid_dim=rows, n=n)
    assert ex.device_status()["code"] == 0
    ex.set_option("row_wait_ms", 0)
    try:
        rows_program(x, w, x, z, grid_dim=rows, n=n)
    finally:
        ex.set_option("row_wait_ms", 4000)
    torch.cuda.synchronize()
    before, plan = ex.launches, ex.build_plan([(rows_program, [x, w, x, want], rows)])
    add, tile = C.vec_add_128, [torch.zeros(128, device="cuda") for _ in range(3)]
    for call in (lambda: rows_program(x, w, x, want, grid_dim=rows, n=n), lambda: add(*tile, grid_dim=1), lambda: plan.run(torch.cuda.current_stream().cuda_stream),
                 lambda: ex.execute_indirect([add], [tile], [0]), lambda: ex.execute_indirect([add], [tile], [0], static_tables=True),
                 lambda: ex.execute_checked(add, C.to_interfaces(tile), 1)):
        with pytest.raises(capi.GintError) as e:
            call()
        assert e.value.status == capi.GINT_ERR_INCOMPLETE
    assert ex.launches == before and ex.device_status(clear=False)["what"] == "a wait gave up" and ex.device_status()["count"] == 1
    assert (z == 9.0).all()
    assert ex.device_status()["code"] == 0
    rows_program(x, w, x, z, grid_dim=rows, n=n)
    assert bits_equal(z.cpu(), want.cpu()) and ex.device_status()["code"] == 0


@pytest.mark.gpu
def test_reading_the_status_waits_for_checked_launches_only():
    """A context that has made no checked launch reads its status without waiting, also while a stream is captured."""
    lib, ctx, status = capi.load_library(), ctypes.c_void_p(), capi.DeviceStatusC()
    assert lib.gint_create(torch.cuda.current_device(), ctypes.byref(ctx)) == 0
    try:
        pd = program(rows=64)
        code = np.ascontiguousarray(np.asarray(pd.program, dtype=np.int32).reshape(-1))
        ti, handle = capi.HTensorInfo(), ctypes.c_uint64()
        fill_tensor_info(ti, pd.input_infos)
        assert lib.gint_program_create(ctx, code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), code.size, ctypes.byref(ti), 4, ctypes.byref(handle)) == 0
        t = [torch.ones(64, 1024, device="cuda") for _ in range(4)]
        graph, bases = torch.cuda.CUDAGraph(), (ctypes.c_uint64 * 8)(*[x.data_ptr() for x in t])
        KEPT.append(graph)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            assert lib.gint_execute(ctx, handle, bases, 4, 64, torch.cuda.current_stream().cuda_stream) == 0
            assert lib.gint_device_status_read(ctx, ctypes.byref(status), 1) == 0 and status.code == 0
        graph.replay()
        torch.cuda.synchronize()
        assert torch.allclose(t[3], torch.ones_like(t[3]))
    finally:
        lib.gint_destroy(ctx)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["bmm4x4", "inv4x4"])
@pytest.mark.parametrize("batch", [1, 31, 33, 64, 1000, 4747, 80001])
def test_lane_programs_give_the_bits_of_the_interpreter(kind, batch):
    """Last tiles of any size, fewer tiles than warps and many rounds of them, ranges, singular and extreme matrices; guard bands."""
    m, ex = _perf_cases(), get_executor()
    g = torch.Generator(device="cuda").manual_seed(batch)
    a, b = torch.randn(batch, 16, device="cuda", generator=g), torch.randn(batch, 16, device="cuda", generator=g)
    a[::5] = 0.0
    a[3::7] *= 1e20
    b[1::9, 3] = float("inf")
    program_, tiles = getattr(m, kind), -(-batch // 32)
    for first, count in ((0, tiles), (tiles // 3, tiles - tiles // 3), (0, (tiles + 1) // 2)):
        def launch():
            buffer = torch.full((batch + 64, 16), 9.0, device="cuda")
            c = buffer[32:32 + batch]
            tensors = [a, b, c] if kind == "bmm4x4" else [a, c]
            ex.execute_range(program_, C.to_interfaces(tensors), first, count, cuda_stream=torch.cuda.current_stream().cuda_stream)
            return [buffer]
        same_bits(launch)
    c = torch.empty_like(a)
    tensors = [a, b, c] if kind == "bmm4x4" else [a, c]
    assert ex.launch_info(program_, C.to_interfaces(tensors), tiles)["form"] == LANES


@pytest.mark.gpu
@pytest.mark.parametrize("batch,tokens,heads,dim", [(1, 1, 1, 128), (2, 37, 3, 64), (1, 6, 2, 33), (2, 12, 3, 80), (1, 31, 2, 96), (3, 50, 7, 127), (2, 333, 5, 128), (4, 1000, 6, 64), (8, 1001, 5, 128)])
@pytest.mark.parametrize("shift", [0, 1])
def test_heads(batch, tokens, heads, dim, shift):
    """The bits of the interpreter: of its tile kernels, or, for rows of 128 at 8-byte boundaries, of its streaming kernel in the vector layout, which
    adds the squares in the same order. Those are also held against the tile kernels' order: one bfloat16 rounding of the 64-bit value, to which sum,
    rsqrt and products in f32 add less than 2^-18. Among the values: rows of zeros, huge and tiny ones, infinities and NaN."""
    ex = get_executor()
    g = torch.Generator(device="cuda").manual_seed(dim)
    count = batch * tokens * heads * dim
    flat = (torch.randn(count + 8, device="cuda", generator=g) * 1.5 + 0.5).bfloat16()
    x = flat[shift:shift + count].view(batch, tokens, heads, dim).transpose(1, 2)
    w = torch.rand(dim + 8, device="cuda", generator=g).bfloat16()[shift:shift + dim]
    total = batch * heads * -(-tokens // 4)
    fours = dim == 128 and shift == 0

    def run(first, n, **options):
        for name, on in options.items():
            ex.set_option(name, on)
        try:
            buffer = torch.full((count + 128,), 9.0, device="cuda").bfloat16()
            y = buffer[64 + shift:64 + shift + count].view(batch, tokens, heads, dim).transpose(1, 2)
            assert (ex.launch_info(heads_program, C.to_interfaces([x, y, w]), total)["form"] == HEADS) == (not options)
            ex.execute_range(heads_program, C.to_interfaces([x, y, w]), first, n, cuda_stream=torch.cuda.current_stream().cuda_stream)
            return buffer.cpu()
        finally:
            for name in options:
                ex.set_option(name, 1)
    for extreme in (False, True):
        if extreme:
            rows = x.reshape(-1, dim).clone()
            for k, v in enumerate((0.0, 1e30, 1e-30, -1e-40, 3e38)):
                rows[k::11] *= v
            for k, v in enumerate((float("inf"), float("-inf"), float("nan"), -0.0)):
                rows[5 + k::13, dim - 1 - k] = v
            flat[shift:shift + count] = rows.view(batch, heads, tokens, dim).transpose(1, 2).reshape(-1)
        for first, n in ((0, total), (total // 3, total - total // 3)):
            got, other = run(first, n), run(first, n, forms=0) if fours else run(first, n, streaming=0)
            assert bits_equal(got, other), mismatch_report(got, other)
            if fours and not extreme:
                tile = run(first, n, streaming=0)
                xd = x.double()
                want = torch.full((count + 128,), 9.0, dtype=torch.float64, device="cuda")
                inside = (tile != 9.0).cuda()
                full = (xd * torch.rsqrt(xd.pow(2).sum(-1, keepdim=True) * 2.0 ** -7 + float(torch.tensor(1e-5).half())) * w.double()).transpose(1, 2).reshape(-1)
                want[64:64 + count] = torch.where(inside[64:64 + count], full, want[64:64 + count])
                torch.testing.assert_close(got.double(), want.cpu(), rtol=2.0 ** -8 + 2.0 ** -18, atol=0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("op", ["fadd", "fmul", "silu", "silu_fmul", "silu_fadd"])
def test_flat_launches_give_the_bits_of_the_interpreter(op, dtype):
    """Lengths around groups, warps' shares and blocks, a group per thread and several, ranges, in place; zeros, infinities and NaN."""
    ex, dt = get_executor(), TYPES[dtype]
    for n, tiles in ((1, 1), (3, 4), (8, 1), (127, 1), (1025, 4), (4096, 1), (40003, 4), (1 << 20, 1), (1212416, 1), (1212421, 4), (5000007, 4)):
        g = torch.Generator(device="cuda").manual_seed(n)
        x, y = [(torch.randn(n, device="cuda", generator=g) * 3).to(dt) for _ in range(2)]
        for k, v in enumerate((0.0, -0.0, float("inf"), float("-inf"), float("nan"), 1e-7, -95.0)):
            x[k + 11:k + 12] = v
        total = -(-n // (128 * tiles))
        kw = {"op": op, "dtype": dtype, "tiles": tiles}
        assert ex.launch_info(flat_program, C.to_interfaces([x, y, torch.empty_like(x)]), total, **kw)["form"] == FLAT
        for first, count in {(0, total), (total // 3, total - total // 3), (0, -(-total // 2))}:
            def launch():
                buffer = torch.full((n + 128,), 9.0, device="cuda").to(dt)
                z, inplace = buffer[64:64 + n], x.clone()
                st = torch.cuda.current_stream().cuda_stream
                ex.execute_range(flat_program, C.to_interfaces([x, y, z]), first, count, cuda_stream=st, **kw)
                ex.execute_range(flat_program, C.to_interfaces([inplace, y, inplace]), first, count, cuda_stream=st, **kw)
                return [buffer, inplace]
            same_bits(launch)
