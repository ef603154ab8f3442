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
        for n, aligned in ((1024, True), (1029, False), (1026, False), (1028, True)):
            slots = [slot(n, elm=2, batch=(rows, n)), slot(n, elm=2, batch=(rows, 1032))]
            r = route(scaled_rows(*HALF, n, 8), slots, count=rows, gather_mask=1)
            assert r == (WIDE_VECTOR if aligned else WIDE), (rows, n, r)
    # without the gather a batch of one row never uses its stride
    assert route(scaled_rows(*HALF, 1029, 8), [slot(1029, elm=2, batch=(1, 1029)), slot(1029, elm=2, batch=(1, 1032))], count=1) == WIDE_VECTOR


def test_a_gathered_f32_row_is_aligned_for_every_index():
    """The 16-byte accesses of the tile kernels rest on the same rule."""
    for rows in (1, 2):
        for stride, aligned in ((1024, True), (1029, False), (1026, False)):
            slots = [slot(1024, batch=(rows, stride)), slot(1024, batch=(rows, 1024))]
            r = route(scaled_rows(*SINGLE, 1024, 8), slots, count=rows, gather_mask=1)
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


@pytest.mark.parametrize("second", [4, 8])
def test_equal_running_values_of_two_loops_are_not_one_value(second):
    """A value that is the same in all four width positions may multiply data in the vector layout. Two loops that add the same terms
    to the same start give the same value only if they run equally often, so a shuffle of both is not such a value."""
    prog = counted(4) + counted(second) + [(O.FShuf2, 0)]      # two positions of each
    for k in range(8):
        prog += [(O.Dup, 0), at(HALF[0], 128 * k, 0), (O.FMul, 0), at(HALF[1], 128 * k, 1)]
    prog += [(O.Pop, 0), (O.Halt, 0)]
    rows = [slot(1024, elm=2, batch=(64, 1024))] * 2
    assert route(prog, rows) == WIDE
    one = counted(4) + [i for k in range(8) for i in ((O.Dup, 0), at(HALF[0], 128 * k, 0), (O.FMul, 0), at(HALF[1], 128 * k, 1))] + [(O.Pop, 0), (O.Halt, 0)]
    assert route(one, rows) == WIDE_VECTOR


@pytest.mark.parametrize("shift,bases,want", [(0, None, WIDE_VECTOR), (128, None, WIDE_VECTOR), (32, None, WIDE), (64, None, WIDE),
                                              (None, 0, WIDE), (None, 64, WIDE), (None, 1 << 20, WIDE_VECTOR)])
def test_what_one_loop_stores_the_same_lanes_load_in_the_next(shift, bases, want):
    """Nothing but a lane's own program order stands between a store of one loop and a load of the next. In the natural layout
    accesses 32 elements apart meet in the same lane, in the vector layout only those 128 apart: by one slot (`shift`) or by two
    slots over one buffer (`bases`: bytes between them)."""
    n_slot, off = (1, shift) if shift is not None else (3, 0)
    prog = [i for k in range(8) for i in (at(HALF[0], 128 * k, 0), at(HALF[1], 128 * k, 1))]
    prog += [i for k in range(4) for i in (at(HALF[0], 128 * k + off, n_slot), (O.FNeg, 0), at(HALF[1], 128 * k, 2))] + [(O.Halt, 0)]
    rows = [slot(1024, elm=2, batch=(64, 1024))] * 4
    addr = [t << 36 for t in range(1, 5)]
    if bases is not None:
        addr[3] = addr[1] + bases
    assert route(prog, rows, bases=addr) == want


@pytest.mark.parametrize("load,elm,want", [(O.LoadGlobal2DTF16, 2, WIDE_VECTOR), (O.LoadGlobal2DTBF16, 2, WIDE_VECTOR), (O.LoadGlobal2DTF32, 4, WIDE),
                                           (O.LoadGlobal2DTU8, 1, WIDE)])
def test_only_sums_of_two_byte_2dt_tiles_change_their_order(load, elm, want):
    """The vector layout adds the elements of 2DT tiles in another order. That is taken for 2-byte elements alone, whose values carry far
    fewer bits than the sum; f32 and u8 sums keep the program's order, as every other sum does."""
    prog = [(O.LoadImm, 0)] + [i for k in range(4) for i in ((load, (32 * k << 4)), (O.Dup, 0), (O.FMul, 0), (O.FAdd, 0))]
    prog += [(O.WarpAllReduceSum, 0)]
    prog += [i for k in range(4) for i in ((O.Dup, 0), (load, (32 * k << 4)), (O.FMul, 0), at(O.StoreGlobal2DTBF16, 32 * k, 1))] + [(O.Pop, 0), (O.Halt, 0)]
    rows = [slot(128, elm=elm, batch=(64, 512), shape2=4, stride2=128), slot(128, elm=2, batch=(64, 512), shape2=4, stride2=128)]
    assert route(prog, rows) == want


@pytest.mark.parametrize("tiles,want", [(4000, WIDE_VECTOR), (12000, 0)])
def test_a_program_too_long_for_the_tile_kernels_has_no_other_route(tiles, want):
    """The tile kernels keep the whole program in shared memory and refuse one that does not fit; whether a launch is refused must not
    depend on addresses, so such a program has no stream with loops either."""
    rows = [slot(128 * tiles, elm=2, batch=(64, 128 * tiles))] * 2
    assert route(scaled_rows(*HALF, 128 * tiles, tiles), rows) == want
