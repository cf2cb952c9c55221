"""Counts whose ids lie on both sides of 2^30, from where on a tile's count of
vertices no longer fits a 32-bit state, or reach the id that pads the engine's
streams (2^31 - 2): totals against the oracle on the same edges with dense ids,
in the same order; shards, which report by rank, refuse the last, and so do
lists whose relabelling would not fit one sort."""
import numpy as np
import pytest

import oracle
import signed_triangle_counting_b200 as stc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top", [(1 << 30) - 1, 1 << 30, (1 << 30) + 5000,
                                 (1 << 31) - 3, (1 << 31) - 2])
def test_ids_around_2_30(top):
    # Vertices in pairs about 2^30 apart, edges among neighbours in a random
    # order of them, and the top id.
    rng = np.random.default_rng(top & 0xFFFF)
    low = rng.integers(0, 4000, 2000)
    ids = np.unique(np.concatenate([low, np.minimum(low + (1 << 30), top), [top - 1, top]]))
    k = len(ids)
    order = rng.permutation(k)
    at = rng.integers(0, k, 60_000)
    a, b = order[at], order[(at + 1 + rng.integers(0, 12, len(at))) % k]
    lo, hi = np.minimum(a, b), np.maximum(a, b)
    sign = np.where((lo * 7 + hi * 13) % 5 < 2, -1, 1).astype(np.int8)
    a, b = np.append(a, k - 1), np.append(b, 0)
    sign = np.append(sign, np.int8(1))
    want = oracle.count_arrays(a.astype(np.uint32), b.astype(np.uint32), sign)
    assert sum(want) > 1000
    with stc.Context(0) as c:
        for persistent in (False, True):
            got = c.count(ids[a].astype(np.uint32), ids[b].astype(np.uint32), sign,
                          persistent=persistent)
            assert got.as_tuple() == want


def test_shard_limit():
    src, dst, sign = np.array([0, 1, 0], np.uint32), np.array([1, 2, 2], np.uint32), np.ones(3, np.int8)
    with stc.Context(0) as c:
        assert sum(c.count_shard(src, dst, sign, 0, 2)[0].as_tuple()) + \
            sum(c.count_shard(src, dst, sign, 1, 2)[0].as_tuple()) == 1
        dst[1] = (1 << 31) - 2
        with pytest.raises(stc.StcError) as e:
            c.count_shard(src, dst, sign, 0, 2)
        assert e.value.status == stc._capi.STC_ERR_LIMIT


def test_relabelled_list_limit():
    import torch
    m = 1 << 31  # self-loops but for one edge with a large id
    src = torch.zeros(m, dtype=torch.int32, device="cuda")
    dst = torch.zeros(m, dtype=torch.int32, device="cuda")
    sign = torch.ones(m, dtype=torch.int8, device="cuda")
    src[0] = -1
    with stc.Context(0) as c:
        with pytest.raises(stc.StcError) as e:
            c.count(src, dst, sign)
        assert e.value.status == stc._capi.STC_ERR_LIMIT
    del src, dst, sign
    torch.cuda.empty_cache()
