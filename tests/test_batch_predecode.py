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
    valid = 0
    for _ in range(300):
        n = int(rng.integers(1, 30))
        code = np.stack([rng.choice([O.LoadGlobal1DF32, O.LoadImm, O.FAdd, O.Dup, O.Pop, O.FPermW, O.DupBroadcastW, O.Swap, O.StoreGlobal1DF32], n),
                         rng.integers(-5, 40, n)], 1).astype(np.int32)
        bad = rng.random(n) < 0.02
        code[bad, 0] = rng.integers(-3, 140, bad.sum())
        if rng.random() < 0.9:
            code[-1] = O.Halt, 0
        valid += check(code, int(rng.integers(1, 9))) > 0
    assert check(np.zeros((0, 2)), 1) < 0 and valid >= 0
