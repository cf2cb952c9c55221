"""A device-side wait that expired (error word 2), set before a call as an
earlier kernel would have: every entry reports STC_ERR_DEVICE_TIMEOUT, and the
context counts rightly again afterwards.  No wait expires for it."""
import ctypes as C

import numpy as np
import pytest

import oracle
import signed_triangle_counting_b200 as stc
from signed_triangle_counting_b200 import _capi

pytestmark = pytest.mark.gpu


def graph(m, seed):
    rng = np.random.default_rng(seed)
    n = m // 6
    src = rng.integers(0, n, m).astype(np.uint32)
    dst = ((src + 1 + rng.integers(0, 30, m)) % n).astype(np.uint32)
    return src, dst, np.where((src + dst) % 3 == 0, -1, 1).astype(np.int8)


def preset(ctx, word):
    f = _capi.lib().stc_test_preset_error
    f.argtypes, f.restype = [C.c_void_p, C.c_uint32], C.c_int
    assert f(ctx._h, word) == 0


def times_out(call):
    with pytest.raises(stc.StcError) as e:
        call()
    assert e.value.status == _capi.STC_ERR_DEVICE_TIMEOUT


@pytest.mark.parametrize("m", [3_000, 700_000])
def test_every_entry_reports_it(m):
    g = graph(m, m)
    want = oracle.count_arrays(*g)
    text = "".join(f"{a} {b} {c}\n" for a, b, c in zip(*(x[:2000].tolist() for x in g))).encode()
    batch = [graph(m // 2, 1), graph(m // 3, 2)]
    each = [oracle.count_arrays(*b) for b in batch]
    big = (g[0].astype(np.uint32) + np.uint32((1 << 32) - m), g[1] + np.uint32((1 << 32) - m), g[2])
    with stc.Context(0) as c:
        csr = c.build_forward_csr(*g)
        calls = [lambda: c.count(*g), lambda: c.count(*g, strategy="merge"),
                 lambda: c.count(*g, persistent=True), lambda: c.count(*big),
                 lambda: c.count(*g, strategy="split"),
                 lambda: c.count_text(text), lambda: c.count_shard(*g, 0, 2),
                 lambda: c.build_forward_csr(*g), lambda: c.count_triangles(csr),
                 lambda: c.count_batch(batch), lambda: c.count_batch(batch, persistent=False)]
        for call in calls:
            preset(c, 2)
            for _ in range(3):  # a batch group is run, capped and captured
                times_out(call)
            preset(c, 0)
            assert c.count(*g).as_tuple() == want
    with stc.Context(0) as c:
        for persistent in (True, True, True, False):
            assert [x.as_tuple() for x in c.count_batch(batch, persistent=persistent)] == each


def test_nothing_is_counted_after_it():
    g = graph(700_000, 7)
    src, dst, sign = (np.ascontiguousarray(x) for x in g)
    n = int(max(src.max(), dst.max())) + 1
    with stc.Context(0) as c:
        for persistent in (False, True):
            assert c.vertex_counts(*g, persistent=persistent).sum() > 0
            buf = np.full(4 * n, 7, np.uint64)
            n_out, o = C.c_uint32(), c._opts(persistent=persistent)
            preset(c, 2)
            rc = _capi.lib().stc_vertex_counts(
                c._h, src.ctypes.data_as(_capi.u32p), dst.ctypes.data_as(_capi.u32p),
                sign.ctypes.data_as(_capi.i8p), len(src), C.byref(o),
                buf.ctypes.data_as(_capi.u64p), len(buf), C.byref(n_out))
            preset(c, 0)
            assert rc == _capi.STC_ERR_DEVICE_TIMEOUT
            assert not buf.any() or (buf == 7).all()
