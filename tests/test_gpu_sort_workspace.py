"""Graphs whose edges and vertices lie on different sides of a sort's tile
limits (606,208 and 2,424,832 keys), in a fresh context each, whose workspace
no larger sort has grown: totals, batches, per-vertex counts and forward CSRs
against the oracle."""
import numpy as np
import pytest

import oracle
import signed_triangle_counting_b200 as stc

pytestmark = pytest.mark.gpu


def graph(n, m, seed):
    rng = np.random.default_rng(seed)
    src = rng.integers(0, n, m).astype(np.uint32)
    dst = ((src + 1 + rng.integers(0, 2, m)) % n).astype(np.uint32)
    src[0], dst[0] = n - 1, 0
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    return src, dst, np.where((lo * 7 + hi * 13) % 3 == 0, -1, 1).astype(np.int8)


@pytest.mark.parametrize("n,m", [(800_000, 500_000), (650_000, 600_000), (1_000_000, 606_208),
                                 (2_500_000, 2_400_000), (4_000_000, 2_424_832)])
def test_more_ids_than_edges(n, m):
    g = graph(n, m, n + m)
    want = oracle.count_arrays(*g)
    assert sum(want) > 0
    with stc.Context(0) as c:
        assert c.count(*g).as_tuple() == want


@pytest.mark.parametrize("n,m", [(400_000, 620_000), (606_208, 606_209), (2_400_000, 2_500_000),
                                 (2_000_000, 3_000_000), (2_424_832, 2_424_833)])
def test_vertices_below_a_limit_edges_above(n, m):
    g = graph(n, m, n + m)
    ref = oracle.ForwardCSR(*g)
    arrays = ref.arrays()
    with stc.Context(0) as c:
        np.testing.assert_array_equal(c.vertex_counts(*g), ref.vertex_counts())
    with stc.Context(0) as c:
        got = c.build_forward_csr(*g)
        for k in ("offsets", "edges", "signs", "fdeg", "rank"):
            np.testing.assert_array_equal(getattr(got, k), arrays[k], err_msg=k)
    parts = [graph(n // 2, m // 2, seed) for seed in (1, 2)]
    want = [oracle.count_arrays(*p) for p in parts]
    with stc.Context(0) as c:
        for persistent in (True, True, True, False):
            assert [x.as_tuple() for x in c.count_batch(parts, persistent=persistent)] == want
