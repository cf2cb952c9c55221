"""The autotuner times its classes on the engine that counts: arcs with a short
list are counted with the head side's keys there too, whatever class is timed,
so a graph of short lists is counted whole by every candidate."""
import ctypes as C

import numpy as np
import pytest

import oracle
from signed_triangle_counting_b200 import _capi

pytestmark = pytest.mark.gpu


def test_short_arcs_are_counted_in_every_class(ctx):
    n = 20_000  # every vertex tied to the next two: triangles (i, i + 1, i + 2)
    src = np.repeat(np.arange(n, dtype=np.uint32), 2)
    dst = ((src + np.tile([1, 2], n)) % n).astype(np.uint32)
    sign = np.where((src + dst) % 3 == 0, -1, 1).astype(np.int8)
    before = ctx.get_tuning()
    try:
        ctx.autotune(src, dst, sign, reps=1)
        out, f = _capi.stc_counts(), _capi.lib().stc_test_counters
        f.argtypes, f.restype = [C.c_void_p, C.POINTER(_capi.stc_counts)], C.c_int
        assert f(ctx._h, C.byref(out)) == 0
    finally:
        ctx.set_tuning(before)
    assert (out.t0, out.t1, out.t2, out.t3) == oracle.count_arrays(src, dst, sign)
