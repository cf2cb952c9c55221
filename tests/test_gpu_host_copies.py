"""Staged copies of pageable host memory at the edges of their 2 MB slots and
256 KB parts, up (edge lists, text, batches of scattered graphs) and down
(edge lists, forward CSRs, per-vertex counts), and host memory that is reused
right after a call."""
import numpy as np
import pytest

import oracle
import signed_triangle_counting_b200 as stc

pytestmark = pytest.mark.gpu


def graph(m, seed):
    rng = np.random.default_rng(seed)
    n = max(4, m // 8)
    src = rng.integers(0, n, m).astype(np.uint32)
    dst = ((src + 1 + rng.integers(0, min(n - 1, 40), m)) % n).astype(np.uint32)
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    return src, dst, np.where((lo * 7 + hi * 13) % 3 == 0, -1, 1).astype(np.int8)


# 4-byte ids: 2^16 fill a part, 2^19 a slot; 8 slots in the ring.
@pytest.mark.parametrize("m", [1, (1 << 16) + 1, (1 << 18) - 1, 1 << 18, (1 << 19) - 1, 1 << 19,
                               (1 << 19) + 1, (9 << 19) + 3])
def test_edge_lists(ctx, m):
    g = graph(m, m)
    want = oracle.count_arrays(*g)
    assert ctx.count(*g).as_tuple() == want
    import torch
    pinned = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).pin_memory().numpy()
              for a in g]
    assert ctx.count(pinned[0].view(np.uint32), pinned[1].view(np.uint32), pinned[2]).as_tuple() == want


def test_memory_reused_after_a_call(ctx):
    a, b = graph(3_000_000, 1), graph(3_000_000, 2)
    want = [oracle.count_arrays(*a), oracle.count_arrays(*b)]
    bufs = [x.copy() for x in a]
    for k in (0, 1, 0, 1):
        for x, y in zip(bufs, (a, b)[k]):
            x[:] = y
        assert ctx.count(*bufs).as_tuple() == want[k]


def test_scattered_batch(ctx):
    sizes = [0, 1, 5, 70_000, 0, 300_000, 3, 524_288, 17, 1_000_003, 2]
    graphs = [graph(m, 50 + i) if m else tuple(np.zeros(0, t) for t in (np.uint32, np.uint32, np.int8))
              for i, m in enumerate(sizes)]
    want = [oracle.count_arrays(*g) if len(g[0]) else (0, 0, 0, 0) for g in graphs]
    got = ctx.count_batch(graphs)
    assert [c.as_tuple() for c in got] == want


@pytest.mark.parametrize("m", [1000, 1 << 19, 1_400_000])
def test_downloads(ctx, m):
    src, dst, sign = graph(m, m + 1)
    text = "".join(f"{a} {b} {c}\n" for a, b, c in zip(src.tolist(), dst.tolist(), sign.tolist()))
    mine, host = ctx.parse_edge_text_gpu(text.encode()), stc.parse_edge_text(text.encode())
    for k in ("src", "dst", "sign"):
        np.testing.assert_array_equal(getattr(mine, k), getattr(host, k))
    csr = ctx.build_forward_csr(src, dst, sign)
    again = ctx.build_forward_csr(dst, src, sign)  # the first one's arrays stay its own
    want = oracle.ForwardCSR(src, dst, sign)
    arrays = want.arrays()
    for c in (csr, again):
        for k in ("offsets", "edges", "signs", "fdeg", "rank"):
            np.testing.assert_array_equal(getattr(c, k), arrays[k], err_msg=k)
    np.testing.assert_array_equal(ctx.vertex_counts(src, dst, sign), want.vertex_counts())


def test_trim_and_use_again():
    g = graph(1_000_000, 9)
    want = oracle.count_arrays(*g)
    with stc.Context(0) as c:
        for _ in range(2):
            assert c.count(*g).as_tuple() == want
            assert stc._capi.lib().stc_ctx_trim(c._h) == 0
