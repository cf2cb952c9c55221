"""A forward CSR given by the caller is checked on the device before any of it
is used as an index: each kind of damage is refused, and the context goes on
counting."""
import numpy as np
import pytest

import oracle
import signed_triangle_counting_b200 as stc
from signed_triangle_counting_b200 import _capi, synth

pytestmark = pytest.mark.gpu


def good():
    el = synth.er(3, 3000, 24_000, 0.6)
    return oracle.ForwardCSR(el.src, el.dst, el.sign)


def broken(kind):
    a = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in good().arrays().items()}
    n, m = a["n"], a["m"]
    if kind == "decrease":
        a["offsets"][n // 2] = a["offsets"][n // 2 - 1] - 1
    elif kind == "past the end":
        a["offsets"][n // 2] = m + 7
    elif kind == "rank twice":
        a["rank"][5] = a["rank"][9]
    elif kind == "rank >= n":
        a["rank"][n - 1] = n
    elif kind == "rank max":
        a["rank"][0] = 0xFFFFFFFF
    elif kind == "id >= n":
        a["edges"][m - 1] = n
    elif kind == "id max":
        a["edges"][0] = 0xFFFFFFFF
    elif kind == "no edges, rank twice":
        a.update(m=0, offsets=np.zeros(n + 1, np.uint64), edges=a["edges"][:0], signs=a["signs"][:0])
        a["rank"][1] = a["rank"][0]
    elif kind == "downhill":
        u = int(np.flatnonzero(np.diff(a["offsets"].astype(np.int64)) > 0)[0])
        a["edges"][int(a["offsets"][u])] = int(np.argmin(a["rank"]))
    return a


@pytest.mark.parametrize("kind", ["decrease", "past the end", "rank twice", "rank >= n", "rank max",
                                  "id >= n", "id max", "no edges, rank twice", "downhill"])
def test_refused(ctx, kind):
    with pytest.raises(stc.StcError) as e:
        ctx.count_triangles(stc.ForwardCSR(**broken(kind)))
    assert e.value.status == _capi.STC_ERR_INVALID_ARGUMENT
    csr = good()
    assert ctx.count_triangles(stc.ForwardCSR(**csr.arrays())).as_tuple() == csr.count()
