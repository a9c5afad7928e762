"""The binding's call module against C functions made by ctypes: the values
that arrive, the handles it takes, and the arguments it leaves to the general
path (None, nothing called)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest


@pytest.fixture(scope="module")
def calls():
    from barbu_gb300 import build
    import os
    if not os.path.exists(build.CALLS):
        build.build_calls()
    from barbu_gb300 import _hscalls
    return _hscalls


class Fake:
    def __init__(self):
        self.seen = []
        self.fns = [C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_float)(self.frame),
                    C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p)(self.floats),
                    C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_uint32)(self.rows)]
        self.f, self.v, self.r = (C.cast(f, C.c_void_p).value for f in self.fns)

    def frame(self, h, dt):
        self.seen.append((h, dt))
        return 7

    def floats(self, h, p):
        self.seen.append((h, p))
        return 0

    def rows(self, h, p, n):
        self.seen.append((h, p, n))
        return -3


def test_calls_pass_values_and_status(calls):
    k, h = Fake(), C.c_void_p(0x1234567812345678)
    a = np.arange(8, dtype=np.float32)
    assert calls.frame(k.f, h, 1.0 / 60.0) == 7
    assert calls.floats(k.v, h, a, 8) == 0
    assert calls.rows(k.r, h, a.reshape(2, 4), 4) == -3
    assert calls.rows(k.r, None, a, 4) == -3
    assert calls.rows(k.r, C.c_void_p(), np.zeros((0, 4), np.float32), 4) == -3
    assert k.seen[0] == (h.value, float(np.float32(1.0 / 60.0)))
    assert k.seen[1:4] == [(h.value, a.ctypes.data), (h.value, a.ctypes.data, 2), (None, a.ctypes.data, 2)]
    assert k.seen[4][0] is None and k.seen[4][2] == 0


@pytest.mark.parametrize("a", [np.zeros(8), np.zeros(7, np.float32), np.zeros(16, np.float32)[::2], [0.0] * 8, None,
                               np.zeros(8, ">f4"), np.zeros(32, np.uint8), np.float32(1.0),
                               np.zeros((4, 2), np.float32).T])
def test_other_arguments_are_left_to_the_general_path(calls, a):
    k, h = Fake(), C.c_void_p(1)
    assert calls.floats(k.v, h, a, 8) is None
    if not (isinstance(a, np.ndarray) and a.dtype == np.float32 and a.flags.c_contiguous and a.size == 8):
        assert calls.rows(k.r, h, a, 8) is None
    for dt in (1, None, "x", np.float32(0.1)):
        assert calls.frame(k.f, h, dt) is None
    for handle in (5, "h", object(), np.zeros(2)):
        assert calls.frame(k.f, handle, 0.1) is None
        assert calls.floats(k.v, handle, np.zeros(8, np.float32), 8) is None
    assert calls.frame(None, h, 0.1) is None and calls.frame(k.f, h) is None
    assert not k.seen
