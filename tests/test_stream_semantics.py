"""A stream with loops computes what its program computes: both are run on symbolic values, the program instruction by instruction,
the stream as the kernels run it -- every instruction of a loop body on U tiles at a time, running values in tile 0."""
import random

import pytest

from gint_b200 import opcodes as O
from gint_b200.host import capi
from test_launch_route import at, descriptors, slot, words

LOOP_BEGIN, REMAP, _, _, ACC_ADD, ACC_FMA, ACC_FMA_SQUARE, SQUARE, MUL_KEEP, SILU, LOOP_END = range(106, 117)
WIDE = 128
MINUS_ZERO = 0x80000000
STEP = {O.LoadGlobal1DF32: 128, O.StoreGlobal1DF32: 128, O.LoadGlobal1DF16: 128, O.StoreGlobal1DF16: 128, O.LoadGlobal2DTF32: 32, O.StoreGlobal2DTF32: 32}
STORES = {O.StoreGlobal1DF32, O.StoreGlobal1DF16, O.StoreGlobal2DTF32}
SIZE = {O.LoadGlobal1DF16: 2, O.StoreGlobal1DF16: 2}


def stream(prog, slots):
    import ctypes
    code, ti = words(prog), descriptors(slots)
    n_max = code.size + 16
    ops, operands = (ctypes.c_int32 * n_max)(), (ctypes.c_uint32 * n_max)()
    n = capi.load_library().gint_debug_transform(code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), code.size, ctypes.byref(ti), len(slots),
                                                 8, 1, ops, operands, n_max)
    assert n >= 0, n
    return list(zip(ops[:n], operands[:n])) or None


_ids = {}


def node(*key):
    """The number of an expression: equal numbers are equal expressions."""
    return _ids.setdefault(key, len(_ids))


def add(a, b):
    zero = node("imm", MINUS_ZERO)
    return b if a == zero else a if b == zero else node("add", *sorted((a, b)))


def mul(a, b):
    return node("mul", *sorted((a, b)))


def fma(t, s1, s2):
    return node("fma", *sorted((t, s1)), s2)


class Machine:
    """Values of tiles as expressions; memory by byte, each byte the (expression, position) last stored there."""

    def __init__(self):
        self.memory = {}

    def access(self, op, operand, value=None):
        t, off, size = operand & 15, operand >> 4, SIZE.get(op, 4)
        cells = [(t, b) for b in range(off * size, (off + STEP[op]) * size, 32)]   # (32 bytes stand for one)
        if value is not None:
            for i, c in enumerate(cells):
                self.memory[c] = (op, value, i)
            return None
        return node("load", op, *(self.memory.get(c, c) for c in cells))

    def step(self, op, operand, st):
        if op in STORES:
            self.access(op, operand, st.pop())
        elif op in STEP:
            st.append(self.access(op, operand))
        elif op == O.LoadImm:
            st.append(node("imm", operand))
        elif op in (O.FAddImm, O.FMulImm, O.FMAImm):
            st.append(node(op, st.pop(), ("operand", operand)))
        elif op in (O.FNeg, O.FExp):
            st.append(node(op, st.pop()))
        elif op == O.FAdd:
            st.append(add(st.pop(), st.pop()))
        elif op == O.FMul:
            st.append(mul(st.pop(), st.pop()))
        elif op in (O.FSub, O.FRSub, O.FDiv, O.FRDiv, O.FGt):
            st.append(node(op, st.pop(), st.pop()))
        elif op == O.FMA:
            st.append(fma(st.pop(), st.pop(), st.pop()))
        elif op == O.Select:
            st.append(node(op, st.pop(), st.pop(), st.pop()))
        elif op == O.Dup:
            st.append(st[-1])
        elif op == O.Dup2:
            st.extend(st[-2:])
        elif op == O.DupX1:
            st.insert(-2, st[-1])
        elif op == O.DupX2:
            st.insert(-3, st[-1])
        elif op == O.Swap:
            st[-1], st[-2] = st[-2], st[-1]
        elif op == O.Pop:
            st.pop()
        elif op == O.Pop2:
            del st[-2:]
        else:
            assert op == O.Nop, op


def run_program(prog):
    m, st = Machine(), []
    for op, operand in prog:
        if op == O.Halt:
            break
        m.step(op, operand, st)
    return st, m.memory


def run_stream(prog, tiles, per_pass):
    """`tiles`: of a flat stream, whose loop has no count of its own."""
    m, st, i = Machine(), [], 0
    while prog[i][0] != O.Halt:
        op, operand = prog[i]
        i += 1
        if op == REMAP:
            continue
        if op != LOOP_BEGIN:
            m.step(op, operand, st)
            continue
        end = next(j for j in range(i, len(prog)) if prog[j][0] == LOOP_END)
        n = operand or tiles
        stacks = [list(st) for _ in range(per_pass)]
        for chunk in range(0, n, per_pass):
            here = range(min(per_pass, n - chunk))
            for op, arg in prog[i:end]:
                if op in (ACC_ADD, ACC_FMA, ACC_FMA_SQUARE):
                    acc = stacks[0][{ACC_ADD: -2, ACC_FMA: -3, ACC_FMA_SQUARE: -2}[op]]
                    for u in here:
                        x = stacks[u]
                        acc = add(x[-1], acc) if op == ACC_ADD else fma(x[-1], x[-1], acc) if op == ACC_FMA_SQUARE else fma(x[-1], x[-2], acc)
                    for x in stacks:
                        del x[{ACC_ADD: -1, ACC_FMA: -2, ACC_FMA_SQUARE: -1}[op]:]
                    stacks[0][-1] = acc
                    continue
                for u in range(per_pass):
                    x = stacks[u]
                    if op >= WIDE:
                        f = op - WIDE
                        if f in STEP and u not in here:    # masked: nothing stored, something loaded
                            x.pop() if f in STORES else x.append(node("masked"))
                        else:
                            m.step(f, arg + ((chunk + u) * STEP[f] << 4) if f in STEP else arg, x)
                    elif op == SQUARE:
                        x.append(mul(x[-1], x.pop()))
                    elif op == MUL_KEEP:
                        x.append(mul(x.pop(), x[-1]))
                    else:
                        assert op == SILU
                        for f, a in ((O.Dup, 0), (O.FNeg, 0), (O.FExp, 0), (O.FAddImm, arg), (O.FRDiv, 0)):
                            m.step(f, a, x)
        st = stacks[0]
        i = end + 1
    return st, m.memory


def check(prog, slots, tiles):
    """True if the program has a stream with loops; it must then compute the same."""
    s = stream(prog, slots)
    if s is None:
        return False
    want = run_program(prog)
    for per_pass in (4, 8):
        got = run_stream(s, tiles, per_pass)
        assert got == want, (per_pass, prog, s)
    return True


def rows(n_slots, n=4096, **kw):
    return [slot(n, batch=(64, n + 1), **kw) for _ in range(n_slots)]


def loop(body, tiles, step=128):
    return [(op, arg + (k * step << 4) if op in STEP else arg) for k in range(tiles) for op, arg in body]


X, Y, OUT = (at(O.LoadGlobal1DF32, 0, t) for t in range(3))
STORE = at(O.StoreGlobal1DF32, 0, 2)


def test_a_row_sum_and_a_scaled_row():
    prog = loop([X, (O.Dup, 0), (O.FMul, 0), (O.FAdd, 0)], 8)
    del prog[3]                                  # the first term starts the sum
    prog += loop([(O.Dup, 0), X, (O.FMul, 0), Y, (O.FMul, 0), STORE], 8) + [(O.Pop, 0), (O.Halt, 0)]
    assert check(prog, rows(3), 8)


def test_a_second_sum_below_the_running_one():
    """(5 + x0) * (y0 + x1 + y1 + ...): the first tile adds into the value below, so it is no tile of the loop."""
    first = [X, (O.FAdd, 0), Y]
    body = [(op, arg + (128 << 4) if op in STEP else arg) for op, arg in [X, (O.FAdd, 0), Y, (O.FAdd, 0)]]
    prog = [(O.LoadImm, 0x40A00000)] + first + loop(body, 7) + [(O.FMul, 0), STORE, (O.Halt, 0)]
    check(prog, rows(3), 8)


def test_a_sum_with_two_terms_per_tile():
    """acc + x0 + y0 + x1 + y1 + ...: the terms keep their order."""
    prog = [(O.LoadImm, 0)] + loop([X, (O.FAdd, 0), Y, (O.FAdd, 0)], 8) + [STORE, (O.Halt, 0)]
    check(prog, rows(3), 8)


@pytest.mark.parametrize("load,store", [(O.LoadGlobal1DF16, O.StoreGlobal1DF32), (O.LoadGlobal1DF32, O.StoreGlobal1DF16)])
def test_a_slot_stored_to_with_another_width(load, store):
    """Tile k of one width covers other elements than tile k of the other: the tiles' loads and stores keep their order."""
    prog = loop([at(load, 0, 0), (O.FAddImm, 0x3F800000), at(store, 0, 0)], 8) + [(O.Halt, 0)]
    check(prog, rows(1), 8)


def test_offsets_that_wrap():
    """The offset of an access has 28 bits: after 2^28 - 128 comes 0, which is no further tile of a loop."""
    def body(k):
        off = ((1 << 28) + 128 * (k - 2)) % (1 << 28)
        return [at(O.LoadGlobal1DF32, off, 0), at(O.StoreGlobal1DF32, off, 1)]
    prog = [x for k in range(4) for x in body(k)] + [(O.Halt, 0)]
    check(prog, rows(2), 4)


def random_body(rng, depth):
    """Instructions with no net effect on the stack that read a few values below it."""
    out, d = [], depth
    for _ in range(rng.randrange(2, 9)):
        choice = [[X], [Y], [at(O.LoadGlobal1DF32, 128, 0)], [(O.LoadImm, rng.randrange(4))]] if d < 4 else []
        if d >= 1:
            choice += [[(O.Dup, 0)], [(O.FMulImm, rng.randrange(4))], [(O.FNeg, 0)], [STORE], [(O.Pop, 0)]]
        if d >= 2:
            choice += [[(op, 0)] for op in (O.FAdd, O.FMul, O.FSub, O.Swap, O.DupX1, O.Dup2, O.FGt)] + [[(O.FAdd, 0)]] * 3
            choice += [[(O.Dup, 0), (O.FMul, 0)], [(O.Dup, 0), X, (O.FMul, 0)], [(O.Dup, 0), Y, (O.Swap, 0), (O.FMul, 0)]]
        if d >= 3:
            choice += [[(op, 0)] for op in (O.FMA, O.Select, O.DupX2)] + [[(O.Dup, 0), (O.FMA, 0)]]
        if d >= 1:
            choice += [[(O.Dup, 0), (O.FNeg, 0), (O.FExp, 0), (O.FAddImm, 0x3F800000), (O.FRDiv, 0)]]
        for ins in rng.choice(choice):
            out.append(ins)
            d += EFFECT[ins[0]]
    while d > depth:
        out.append((rng.choice((O.FAdd, O.Pop)), 0) if d >= 2 else (O.Pop, 0))
        d -= 1
    while d < depth:
        out.append(X)
        d += 1
    return out


EFFECT = {O.LoadGlobal1DF32: 1, O.StoreGlobal1DF32: -1, O.LoadImm: 1, O.Dup: 1, O.FMulImm: 0, O.FNeg: 0, O.Pop: -1, O.FAdd: -1, O.FMul: -1, O.FSub: -1,
          O.Swap: 0, O.DupX1: 1, O.Dup2: 2, O.FGt: -1, O.FMA: -2, O.Select: -2, O.DupX2: 1, O.FExp: 0, O.FAddImm: 0, O.FRDiv: -1}


@pytest.mark.parametrize("seed", range(60))
def test_random_loops(seed):
    """Bodies repeated over tiles, some behind a first tile whose last instructions are missing, at several stack depths."""
    rng, streams = random.Random(seed), 0
    for _ in range(120):
        depth, tiles = rng.randrange(4), rng.randrange(2, 12)
        prog = [(O.LoadImm, 100 + k) for k in range(depth)]
        for _ in range(rng.randrange(1, 3)):
            body = random_body(rng, depth)
            whole = loop(body, tiles)
            cut = rng.choice((0, 0, 1, 2))
            lost = body[len(body) - cut:]
            if cut and body[-1][0] == O.FAdd and depth + 1 <= 4 and sum(EFFECT[op] for op, _ in lost) < 0:
                d0 = depth - sum(EFFECT[op] for op, _ in body[:len(body) - cut])
                if d0 < 0 or d0 > depth:
                    continue
                whole = whole[:len(body) - cut] + whole[len(body):]
                prog += whole + [(O.Pop, 0)] * (-sum(EFFECT[op] for op, _ in lost))
            else:
                prog += whole
        prog.append((O.Halt, 0))
        d, ok = 0, True
        for op, _ in prog[:-1]:
            need = {O.FMA: 3, O.Select: 3, O.DupX2: 3}.get(op, 2 if op in (O.FAdd, O.FMul, O.FSub, O.Swap, O.DupX1, O.Dup2, O.FGt, O.FRDiv) else
                                                           0 if op in (O.LoadGlobal1DF32, O.LoadImm) else 1)
            ok = ok and d >= need
            d += EFFECT[op]
            ok = ok and d <= 8
        if ok:
            streams += check(prog, rows(3), tiles)
    assert streams >= 5
