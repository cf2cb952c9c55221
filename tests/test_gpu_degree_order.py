"""The totals build's vertex order (sampled degrees, hubs counted apart, ranks
from 8-bit degree steps) where it can go wrong: every degree step, rank tiles
of 4,096 vertices, hubs above and below the sample's threshold, ids past 2^24
and batches of more graphs than one digit.  Counts against the oracle, whose
order is the reference's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def signs(src, dst):
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    return np.where((lo * 7 + hi * 13) % 5 < 2, -1, 1).astype(np.int8)


def check(ctx, src, dst, n_triangles_min=1):
    src, dst = src.astype(np.uint32), dst.astype(np.uint32)
    sg = signs(src, dst)
    want = oracle.count_arrays(src, dst, sg)
    assert sum(want) >= n_triangles_min
    assert ctx.count(src, dst, sg).as_tuple() == want


@pytest.mark.parametrize("n", [3, 4095, 4096, 4097, 8193, 20_000])
def test_rank_tiles(ctx, n):
    # A wheel: every rim vertex has degree 3, the hub n - 1.
    rim = np.arange(1, n)
    check(ctx, np.concatenate([rim, rim]), np.concatenate([np.zeros(n - 1, int), np.roll(rim, 1)]))


def test_every_degree_step(ctx):
    # Fans with 1 .. 2^17 triangles: a vertex in (nearly) every degree step.
    src, dst, at = [], [], 0
    for k in sorted({max(1, int(2 ** (e / 8))) for e in range(17 * 8 + 1)}):
        spokes = np.arange(at + 1, at + 2 + k)
        src += [np.full(k + 1, at), spokes[:-1]]
        dst += [spokes, spokes[1:]]
        at += k + 2
    check(ctx, np.concatenate(src), np.concatenate(dst))


@pytest.mark.parametrize("m", [(1 << 20) - 1, 1 << 20, 3_000_001])
def test_hubs(ctx, m):
    # Half of the edges meet one of nine hubs, in random order and direction.
    rng = np.random.default_rng(m)
    n = m // 4
    a = rng.integers(0, n, m)
    b = np.where(rng.random(m) < 0.5, rng.integers(0, 9, m) * (n // 9), (a + 1 + rng.integers(0, 50, m)) % n)
    swap = rng.random(m) < 0.5
    check(ctx, np.where(swap, a, b), np.where(swap, b, a))


@pytest.mark.parametrize("top", [(1 << 24) + 5, (1 << 25) + 9])
def test_sparse_large_id_space(ctx, top):
    rng = np.random.default_rng(top)
    a = rng.integers(0, 3000, 60_000) * (top // 3000)
    b = rng.integers(0, 3000, 60_000) * (top // 3000)
    check(ctx, np.append(a, top - 1), np.append(b, 0))


@pytest.mark.parametrize("G", [1, 2, 255, 256, 257, 700])
def test_many_small_graphs(ctx, G):
    rng = np.random.default_rng(G)
    graphs = []
    for g in range(G):
        k = 3 + g % 9
        a, b = np.triu_indices(k, 1)
        p = rng.permutation(k + 2).astype(np.uint32)
        graphs.append((p[a], p[b], signs(p[a], p[b])))
    want = [oracle.count_arrays(*x) for x in graphs]
    for persistent in (True, True, False):
        got = ctx.count_batch(graphs, persistent=persistent)
        assert [c.as_tuple() for c in got] == want
