"""Lists that native code converts: the same calls and results as the conversion in Python, on the CPU (the native step is a recording stand-in)."""
import ctypes
import os
import random
import shutil
import sysconfig

import numpy as np
import pytest

from llama_cpp import _cabi
from llama_cpp.engine import LayeredEngine, int32s

pytestmark = pytest.mark.skipif(_cabi.load_lists() is None, reason="built without Python's headers")

STEP = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int32),
                        ctypes.POINTER(ctypes.c_int32), ctypes.c_int, ctypes.c_void_p, ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int32))


class Recorder:
    """b2_step that writes down its arguments; token 7 + entry for all that sample, logits of row r are r."""

    def __init__(self, V):
        self.calls, self.V = [], V
        self.b2_step = self._step
        self.native = STEP(self._step)

    def _step(self, h, n, slots, counts, tokens, rows, n_want, logits, flags, out):
        c = [counts[i] for i in range(n)]
        r = [rows[i] for i in range(n_want)] if n_want else []
        self.calls.append(([slots[i] for i in range(n)], c, [tokens[i] for i in range(sum(c))], r, [flags[i] for i in range(n)]))
        address = logits if isinstance(logits, int) else getattr(logits, "value", None)
        for i, x in enumerate(r):
            np.ctypeslib.as_array((ctypes.c_float * self.V).from_address(address + 4 * self.V * i))[:] = x
        for i in range(n):
            out[i] = 7 + i if flags[i] else -1
        return 0


def engine(native, V=5, room=64):
    eng = LayeredEngine.__new__(LayeredEngine)
    eng.lib, eng._h, eng.max_step_tokens = Recorder(V), None, room
    eng.dims = type("Dims", (), {"n_vocab": V})
    eng._lists = _cabi.load_lists() if native else None
    eng._step = ctypes.cast(eng.lib.native, ctypes.c_void_p).value
    return eng


@pytest.mark.parametrize("seed", range(30))
def test_same_calls_and_results(seed):
    rng = random.Random(seed)
    n = rng.choice([1, 2, 5, 64, 65])
    entries = [(rng.randrange(100), [rng.randrange(-3, 9) for _ in range(rng.choice([1, 1, 2, 30]))]) for _ in range(n)]
    want = rng.choice([None, [[j for j in range(len(t)) if rng.random() < .3] for _, t in entries]])
    sample = rng.choice([None, [rng.random() < .5 for _ in entries]])
    if seed % 5 == 0:                                          # forms that are not plain lists
        entries = tuple((s, tuple(t)) if rng.random() < .5 else [s, np.array(t)] for s, t in entries)
    if seed % 7 == 0 and sample:
        sample = [int(f) for f in sample]
    engines = [engine(True), engine(False)]
    (lg, got), (ref, expect) = [e.step(entries, want=want, sample=sample) for e in engines]
    assert engines[0].lib.calls == engines[1].lib.calls and got == expect and np.array_equal(lg, ref) and lg.shape == ref.shape


@pytest.mark.parametrize("entries,want", [([(0, [])], None), ([(0, [1])], [[1]]), ([(0, [2 ** 40])], None), ([(0, [1.5])], None), ([], None)])
def test_what_is_no_step_is_left_to_the_general_path(entries, want):
    outcomes = []
    for native in (True, False):
        eng = engine(native)
        try:
            outcomes.append((eng.step(entries, want=want)[1], eng.lib.calls))
        except Exception as e:
            outcomes.append(type(e))
    assert outcomes[0] == outcomes[1]


def test_int_arrays():
    for values in ([], [3] * 12, list(range(-20, 20)), tuple(range(40)), [2 ** 31 - 1, -2 ** 31] * 8, [np.int64(3)] * 20, [True] * 13, range(30), np.arange(20)):
        assert list(int32s(values)) == [int(v) for v in values]
    assert list(int32s([2 ** 32 + 5] * 20)) == [5] * 20        # (ctypes keeps the low bits; the engine then checks the range)


def load_from(folder, monkeypatch):
    monkeypatch.setattr(_cabi, "LIB_PATH", str(folder / "libb200gguf.so"))
    monkeypatch.setattr(_cabi, "_lists", False)
    return _cabi.load_lists()


def test_a_library_of_another_interpreter_is_not_loaded(tmp_path, monkeypatch):
    """What it compiled in of CPython's objects holds for the interpreter whose headers it was built with."""
    built = [f for f in os.listdir(os.path.dirname(_cabi.LIB_PATH)) if f.startswith("libb200_pylists") and sysconfig.get_config_var("SOABI") in f]
    assert len(built) == 1
    whole = os.path.join(os.path.dirname(_cabi.LIB_PATH), built[0])
    for name in ("libb200_pylists.so", "libb200_pylists.cpython-39-x86_64-linux-gnu.so"):
        shutil.copy(whole, tmp_path / name)
    assert load_from(tmp_path, monkeypatch) is None
    shutil.copy(whole, tmp_path / built[0])
    assert load_from(tmp_path, monkeypatch) is not None


def test_a_library_that_does_not_load_is_none(tmp_path, monkeypatch):
    (tmp_path / ("libb200_pylists" + sysconfig.get_config_var("EXT_SUFFIX"))).write_bytes(b"not a library")
    assert load_from(tmp_path, monkeypatch) is None
    assert list(int32s(list(range(30)))) == list(range(30))
