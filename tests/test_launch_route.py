"""Which kernels a launch runs on, asked of the library without a device (gint_debug_route): every condition that a fast or a
reordered stream rests on has to hold for the launch's own addresses and options."""
import ctypes
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

from gint_b200 import opcodes as O  # noqa: E402
from gint_b200.host import capi  # noqa: E402

EARLY, WIDE, WIDE_VECTOR, FLAT = 1, 1 << 4, 2 << 4, 1 << 6


def slot(shape1, stride1=1, elm=4, batch=(1, 0), grid1=1, step1=0, shape2=1, stride2=0):
    """One tensor slot: (shape1, stride1, elm_size, (batch shape, stride), grid dim 1, grid step 1, shape2, stride2)."""
    return shape1, stride1, elm, batch, grid1, step1, shape2, stride2


def descriptors(slots):
    ti = capi.HTensorInfo()
    for t, (shape1, stride1, elm, batch, grid1, step1, shape2, stride2) in enumerate(slots):
        ti.elm_size[t] = elm
        for j in range(4):
            ti.batch_shape[t][j], ti.batch_strides[t][j] = (batch if j == 0 else (1, 0))
        ti.block_shape_stride_1[t][0], ti.block_shape_stride_1[t][1] = shape1, stride1
        ti.block_shape_stride_2[t][0], ti.block_shape_stride_2[t][1] = shape2, stride2
        ti.block_grid_dims[t][0], ti.block_grid_dims[t][1] = grid1, 1
        ti.block_grid_steps[t][0], ti.block_grid_steps[t][1] = step1, 0
    return ti


def words(prog):
    return np.array([[op, operand & 0xFFFFFFFF] for op, operand in prog], dtype=np.uint32).view(np.int32).reshape(-1)


def route(prog, slots, bases=None, first=0, count=64, gather_mask=0, gather_extent=1 << 30):
    code, ti, n = words(prog), descriptors(slots), len(slots)
    addr = (ctypes.c_uint64 * 8)(*(bases or [(t + 1) << 36 for t in range(n)]))
    r = capi.load_library().gint_debug_route(code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), code.size, ctypes.byref(ti), n, addr, first, count,
                                             gather_mask, gather_extent)
    assert r >= 0, r
    return r


def at(op, off, t):
    return op, (off << 4) | t


HALF = (O.LoadGlobal1DF16, O.StoreGlobal1DF16)
SINGLE = (O.LoadGlobal1DF32, O.StoreGlobal1DF32)


def scaled_rows(load, store, n, tiles):
    """out = 2 * x, one row per logical program."""
    p = []
    for k in range(tiles):
        p += [at(load, 128 * k, 0), (O.FMulImm, 0x40000000), at(store, 128 * k, 1)]
    return p + [(O.Halt, 0)]


def test_a_gathered_row_is_aligned_for_every_index():
    """A gathered launch multiplies the row index with the batch stride also where the batch has one row, so 4-element accesses need
    a stride of whole groups of 4 elements there too (an odd row of an odd stride starts at any byte)."""
    for rows in (1, 2):
        for n, aligned in ((2048, True), (2053, False), (2050, False), (2052, True)):
            slots = [slot(n, elm=2, batch=(rows, n)), slot(n, elm=2, batch=(rows, 2056))]
            r = route(scaled_rows(*HALF, n, 16), slots, count=rows, gather_mask=1)
            assert r == (WIDE_VECTOR if aligned else WIDE), (rows, n, r)
    # without the gather a batch of one row never uses its stride
    assert route(scaled_rows(*HALF, 2053, 16), [slot(2053, elm=2, batch=(1, 2053)), slot(2053, elm=2, batch=(1, 2056))], count=1) == WIDE_VECTOR


def test_a_gathered_f32_row_is_aligned_for_every_index():
    """The 16-byte accesses of the tile kernels rest on the same rule."""
    for rows in (1, 2):
        for stride, aligned in ((2048, True), (2053, False), (2050, False)):
            slots = [slot(2048, batch=(rows, stride)), slot(2048, batch=(rows, 2048))]
            r = route(scaled_rows(*SINGLE, 2048, 16), slots, count=rows, gather_mask=1)
            assert (r == EARLY) == aligned and r != WIDE_VECTOR, (rows, stride, r)


def test_gathered_matrix_rows_are_aligned_for_every_index():
    """... and so do 2DW rows and staged row blocks."""
    prog = [at(O.LoadGlobal2DWF32, 0, 0), at(O.StoreGlobal2DWF32, 0, 1), (O.Halt, 0)]
    for stride, aligned in ((128, True), (129, False)):
        slots = [slot(32, 4, batch=(1, stride), shape2=4, stride2=1), slot(32, 4, batch=(1, 128), shape2=4, stride2=1)]
        r = route(prog, slots, count=1, gather_mask=1)
        assert (r == EARLY) == aligned, (stride, r)


def test_a_flat_loop_stays_below_31_bits():
    """A flat launch counts elements through the whole grid, and the offset written in the program comes on top: the sum has to fit an
    int, or a masked access far behind the tensor becomes an unmasked one in front of it."""
    n_programs = 15_000_000
    for off in (0, 128, (1 << 28) - 128):
        prog = [at(O.LoadGlobal1DF32, off, 0), at(O.StoreGlobal1DF32, off, 1), (O.Halt, 0)]
        slots = [slot(100000, grid1=n_programs, step1=128)] * 2
        r = route(prog, slots, count=n_programs)
        assert bool(r & FLAT) == (n_programs * 128 + off < (1 << 31) - 8192), (off, r)


def counted(tiles):
    """A running value that counts the tiles of a copy loop."""
    return [(O.LoadImm, 0)] + [i for k in range(tiles) for i in (at(HALF[0], 128 * k, 0), at(HALF[1], 128 * k, 1), (O.LoadImm, 0x3F800000), (O.FAdd, 0))]


@pytest.mark.parametrize("second", [8, 16])
def test_equal_running_values_of_two_loops_are_not_one_value(second):
    """A value that is the same in all four width positions may multiply data in the vector layout. Two loops that add the same terms
    to the same start give the same value only if they run equally often, so a shuffle of both is not such a value."""
    prog = counted(8) + counted(second) + [(O.FShuf2, 0)]      # two positions of each
    for k in range(16):
        prog += [(O.Dup, 0), at(HALF[0], 128 * k, 0), (O.FMul, 0), at(HALF[1], 128 * k, 1)]
    prog += [(O.Pop, 0), (O.Halt, 0)]
    rows = [slot(2048, elm=2, batch=(64, 2048))] * 2
    assert route(prog, rows) == WIDE
    one = counted(8) + [i for k in range(16) for i in ((O.Dup, 0), at(HALF[0], 128 * k, 0), (O.FMul, 0), at(HALF[1], 128 * k, 1))] + [(O.Pop, 0), (O.Halt, 0)]
    assert route(one, rows) == WIDE_VECTOR


@pytest.mark.parametrize("shift,bases,want", [(0, None, WIDE_VECTOR), (128, None, WIDE_VECTOR), (32, None, WIDE), (64, None, WIDE),
                                              (None, 0, WIDE), (None, 64, WIDE), (None, 1 << 20, WIDE_VECTOR)])
def test_what_one_loop_stores_the_same_lanes_load_in_the_next(shift, bases, want):
    """Nothing but a lane's own program order stands between a store of one loop and a load of the next. In the natural layout
    accesses 32 elements apart meet in the same lane, in the vector layout only those 128 apart: by one slot (`shift`) or by two
    slots over one buffer (`bases`: bytes between them)."""
    n_slot, off = (1, shift) if shift is not None else (3, 0)
    prog = [i for k in range(16) for i in (at(HALF[0], 128 * k, 0), at(HALF[1], 128 * k, 1))]
    prog += [i for k in range(4) for i in (at(HALF[0], 128 * k + off, n_slot), (O.FNeg, 0), at(HALF[1], 128 * k, 2))] + [(O.Halt, 0)]
    rows = [slot(2048, elm=2, batch=(64, 2048))] * 4
    addr = [t << 36 for t in range(1, 5)]
    if bases is not None:
        addr[3] = addr[1] + bases
    assert route(prog, rows, bases=addr) == want


@pytest.mark.parametrize("load,elm,want", [(O.LoadGlobal2DTF16, 2, WIDE_VECTOR), (O.LoadGlobal2DTBF16, 2, WIDE_VECTOR), (O.LoadGlobal2DTF32, 4, WIDE),
                                           (O.LoadGlobal2DTU8, 1, WIDE)])
def test_only_sums_of_two_byte_2dt_tiles_change_their_order(load, elm, want):
    """The vector layout adds the elements of 2DT tiles in another order. That is taken for 2-byte elements alone, whose values carry far
    fewer bits than the sum; f32 and u8 sums keep the program's order, as every other sum does."""
    prog = [(O.LoadImm, 0)] + [i for k in range(12) for i in ((load, (32 * k << 4)), (O.Dup, 0), (O.FMul, 0), (O.FAdd, 0))]
    prog += [(O.WarpAllReduceSum, 0)]
    prog += [i for k in range(12) for i in ((O.Dup, 0), (load, (32 * k << 4)), (O.FMul, 0), at(O.StoreGlobal2DTBF16, 32 * k, 1))] + [(O.Pop, 0), (O.Halt, 0)]
    rows = [slot(384, elm=elm, batch=(64, 1536), shape2=4, stride2=384), slot(384, elm=2, batch=(64, 1536), shape2=4, stride2=384)]
    assert route(prog, rows) == want


@pytest.mark.parametrize("tiles,want", [(4000, WIDE_VECTOR), (12000, 0)])
def test_a_program_too_long_for_the_tile_kernels_has_no_other_route(tiles, want):
    """The tile kernels keep the whole program in shared memory and refuse one that does not fit; whether a launch is refused must not
    depend on addresses, so such a program has no stream with loops either."""
    rows = [slot(128 * tiles, elm=2, batch=(64, 128 * tiles))] * 2
    assert route(scaled_rows(*HALF, 128 * tiles, tiles), rows) == want


def normalised_rows(load, store, tiles, step=128):
    """out = x * sum(x): every row loaded twice."""
    p = [(O.LoadImm, 0)] + [i for k in range(tiles) for i in (at(load, step * k, 0), (O.FAdd, 0))] + [(O.WarpAllReduceSum, 0)]
    if step == 128:      # ... and over the four width values
        p += [(O.Dup, 0), (O.FPermW, 0x01000302), (O.FAdd, 0), (O.Dup, 0), (O.FPermW, 0x02030001), (O.FAdd, 0)]
    return p + [i for k in range(tiles) for i in ((O.Dup, 0), at(load, step * k, 0), (O.FMul, 0), at(store, step * k, 1))] + [(O.Pop, 0), (O.Halt, 0)]


@pytest.mark.parametrize("tiles,rows,want", [(2, 1184, WIDE), (2, 1185, 0), (3, 9472, WIDE), (3, 9473, 0), (4, 59200, WIDE), (4, 59201, 0), (5, 200000, WIDE)])
def test_short_f32_rows_stream_only_in_small_launches(tiles, rows, want):
    """Both sides of the lines: unaligned f32 rows that are loaded twice."""
    n = 128 * tiles - 3
    r = route(normalised_rows(*SINGLE, tiles), [slot(n, batch=(rows, n))] * 2, count=rows)
    assert r & (WIDE | WIDE_VECTOR) == want, r


@pytest.mark.parametrize("form,tiles,n,rows,want", [("once", 15, 1917, 100, 0), ("once", 16, 2045, 1184, WIDE), ("once", 16, 2045, 1185, 0), ("twice", 16, 2048, 100, 0)])
def test_f32_rows_loaded_once_stream_only_where_long_and_few(form, tiles, n, rows, want):
    prog = scaled_rows(*SINGLE, n, tiles) if form == "once" else normalised_rows(*SINGLE, tiles)      # (the last: aligned rows of whole tiles)
    assert route(prog, [slot(n, batch=(rows, n))] * 2, count=rows) & (WIDE | WIDE_VECTOR) == want


@pytest.mark.parametrize("tiles,aligned,rows,want", [(4, True, 9, WIDE_VECTOR), (5, True, 9, 0), (8, True, 90000, WIDE_VECTOR), (10, True, 1184, WIDE_VECTOR), (10, True, 1185, 0),
                                                     (11, True, 90000, WIDE_VECTOR), (10, False, 9, 0), (11, False, 1184, WIDE), (11, False, 1185, 0), (16, False, 90000, WIDE)])
def test_half_precision_rows(tiles, aligned, rows, want):
    n = 128 * tiles - (0 if aligned else 1)
    assert route(normalised_rows(*HALF, tiles), [slot(n, elm=2, batch=(rows, n))] * 2, count=rows) & (WIDE | WIDE_VECTOR) == want


@pytest.mark.parametrize("load,store,elm,tiles,aligned,want", [
    (O.LoadGlobal2DTBF16, O.StoreGlobal2DTBF16, 2, 3, True, 0), (O.LoadGlobal2DTBF16, O.StoreGlobal2DTBF16, 2, 4, True, WIDE_VECTOR),
    (O.LoadGlobal2DTBF16, O.StoreGlobal2DTBF16, 2, 5, False, 0), (O.LoadGlobal2DTBF16, O.StoreGlobal2DTBF16, 2, 6, False, WIDE),
    (O.LoadGlobal2DTF16, O.StoreGlobal2DTF16, 2, 9, False, 0), (O.LoadGlobal2DTF16, O.StoreGlobal2DTF16, 2, 10, False, WIDE),
    (O.LoadGlobal2DTF32, O.StoreGlobal2DTF32, 4, 5, True, 0), (O.LoadGlobal2DTF32, O.StoreGlobal2DTF32, 4, 6, True, WIDE)])
def test_2dt_rows(load, store, elm, tiles, aligned, want):
    n = 32 * tiles - (0 if aligned else 1)
    slots = [slot(n, elm=elm, batch=(64, 4 * n), shape2=4, stride2=n)] * 2
    assert route(normalised_rows(load, store, tiles, 32), slots) & (WIDE | WIDE_VECTOR) == want


@pytest.mark.parametrize("load,store,elm,math,whole,n,want", [
    (*SINGLE, 4, False, False, 1 << 22, 0), (*SINGLE, 4, False, False, (1 << 22) + 128, FLAT), (*SINGLE, 4, True, False, 1 << 25, 0),
    (*SINGLE, 4, False, True, 1 << 23, 0), (*SINGLE, 4, False, True, (1 << 23) + 128, FLAT), (*HALF, 2, True, True, 1 << 21, 0), (*HALF, 2, True, True, (1 << 21) + 128, FLAT),
    (HALF[0], SINGLE[1], 2, True, True, 1 << 22, 0), (HALF[0], SINGLE[1], 2, True, True, (1 << 22) + 128, FLAT)])
def test_flat_programs(load, store, elm, math, whole, n, want):
    prog = [at(load, 0, 0), (O.FSqrt, 0) if math else (O.FNeg, 0), at(store, 0, 1), (O.Halt, 0)]
    length = n if whole else n - 1
    slots = [slot(length, elm=elm, grid1=n // 128, step1=128), slot(length, elm=4 if store == SINGLE[1] else elm, grid1=n // 128, step1=128)]
    assert route(prog, slots, count=n // 128) & FLAT == want
