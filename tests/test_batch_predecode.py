"""The one-pass pre-decoder of candidate batches: the stream and the status of the general one, for recorded, random and malformed programs."""
import ctypes

import numpy as np
import pytest

from gint_b200 import opcodes as O
from gint_b200.host import capi
from gint_b200.programs import load_records, recorded

DIFFERS = -(1 << 31)


def check(code, n_tensors):
    code = np.ascontiguousarray(np.asarray(code, dtype=np.int32).reshape(-1))
    r = capi.load_library().gint_debug_predecode_batch(code.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), int(code.size), n_tensors, None, 0)
    assert r != DIFFERS, code[:40]
    return r


def test_recorded_programs():
    for name in load_records():
        rec = recorded(name)
        r = check(rec.bytecode, len(rec.tensor_infos))
        assert (r > 0) == (name != "execute_everything")


@pytest.mark.parametrize("seed", range(20))
def test_random_words(seed):
    """Mostly invalid programs: every error in its place, opcodes beyond the table, negative ones, slots out of range, no Halt."""
    rng = np.random.default_rng(seed)
    effects = {O.LoadGlobal1DF32: (0, 1), O.LoadImm: (0, 1), O.FAdd: (2, -1), O.Dup: (1, 1), O.Pop: (1, -1), O.FPermW: (1, 0), O.DupBroadcastW: (1, 1),
               O.Swap: (2, 0), O.StoreGlobal1DF32: (1, -1)}
    valid = broken = 0
    for _ in range(300):
        ops, depth = [], 0
        for _ in range(int(rng.integers(1, 30))):     # correct as far as the stack goes, slots out of range now and then
            op = rng.choice([op for op, (need, net) in effects.items() if depth >= need and depth + net <= 8])
            ops.append(op)
            depth += effects[op][1]
        slots = rng.integers(0, 8 if rng.random() < 0.1 else 4, len(ops))
        code = np.stack([ops, np.where([op in (O.LoadGlobal1DF32, O.StoreGlobal1DF32) for op in ops], (rng.integers(0, 40, len(ops)) << 4) | slots,
                                       rng.integers(-5, 40, len(ops)))], 1).astype(np.int32)
        if rng.random() < 0.5:                        # then spoilt
            bad = rng.random(len(ops)) < 0.05
            code[bad, 0] = rng.choice([*effects, -3, 106, 139], bad.sum())
        if rng.random() < 0.9:
            code = np.concatenate([code, [[O.Halt, 0]]]).astype(np.int32)
        r = check(code, 4)
        valid, broken = valid + (r > 0), broken + (r < 0)
    assert valid > 50 and broken > 20
    assert check(np.zeros((0, 2)), 1) < 0
