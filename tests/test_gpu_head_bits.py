"""The head side's bitmap classes (heads with more than 32 out-neighbours whose
later ranks span at most 2^16, or more than 128 and at most 2^18): extents at
every chunk remainder, lists at the class edges, several graphs in one union,
and ranks on both sides of both windows, against the oracle or the tail
side's strategies."""
import numpy as np
import pytest

import oracle
import signed_triangle_counting_b200 as stc

pytestmark = pytest.mark.gpu


def clique_with_fringe(k, fringe, seed):
    """K_k with random signs, plus `fringe` vertices tied to random clique
    members (they shift the lists' positions and add short in-lists)."""
    rng = np.random.default_rng(seed)
    a, b = np.triu_indices(k, 1)
    fa = np.repeat(np.arange(k, k + fringe), 3)
    fb = rng.integers(0, k, len(fa))
    perm = rng.permutation(k + fringe).astype(np.uint32)
    src, dst = perm[np.concatenate([a, fa])], perm[np.concatenate([b, fb])]
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    h = (lo * 2654435761 ^ hi * 40503) >> 7  # duplicates agree in sign
    return src, dst, np.where(h % 5 < 3, 1, -1).astype(np.int8)


@pytest.mark.parametrize("k,fringe", [(33, 0), (34, 3), (35, 40), (66, 2), (129, 0), (130, 1), (131, 5), (137, 64), (160, 333),
                                      (257, 2), (1030, 7), (1300, 1111)])
def test_clique_sizes(ctx, k, fringe):
    g = clique_with_fringe(k, fringe, k)
    want = oracle.count_arrays(*g)
    for strategy in ("auto", "head"):
        assert ctx.count(*g, strategy=strategy).as_tuple() == want
        assert ctx.count(*g, strategy=strategy, persistent=True).as_tuple() == want


def test_union_of_graphs(ctx):
    graphs = [clique_with_fringe(k, f, 7 * k) for k, f in ((140, 3), (3, 0), (200, 50), (135, 9))]
    want = [oracle.count_arrays(*g) for g in graphs]
    for persistent in (True, False):
        got = ctx.count_batch(graphs, persistent=persistent)
        assert [c.as_tuple() for c in got] == want


def test_both_sides_of_the_windows(ctx):
    import torch
    # Uniform random: out-degrees around 140 at every rank, and 2^18 + 20,000
    # vertices, so heads lie inside and below the windows.
    n, m = (1 << 18) + 20_000, 40_000_000
    gen = torch.Generator(device="cuda").manual_seed(5)
    src, dst = (torch.randint(0, n, (m,), dtype=torch.int32, device="cuda", generator=gen)
                for _ in range(2))
    sign = (((src ^ dst) & 7) < 3).to(torch.int8) * -2 + 1  # duplicates agree in sign
    torch.cuda.synchronize()
    want = ctx.count(src, dst, sign, strategy="hash").as_tuple()
    assert sum(want) > 3_000_000
    for strategy in ("auto", "head"):
        assert ctx.count(src, dst, sign, strategy=strategy).as_tuple() == want


@pytest.mark.parametrize("k,fringe", [(9, 4), (33, 0), (36, 7), (130, 1), (140, 200), (300, 33)])
def test_vertex_counts_of_cliques(ctx, k, fringe):
    g = clique_with_fringe(k, fringe, 3 * k)
    want = oracle.ForwardCSR(*g).vertex_counts()
    for persistent in (False, True):
        np.testing.assert_array_equal(ctx.vertex_counts(*g, persistent=persistent), want)


def test_vertex_counts_both_sides_of_the_windows(ctx):
    rng = np.random.default_rng(11)
    n, m = (1 << 18) + 20_000, 36_000_000
    src, dst = (rng.integers(0, n, m, dtype=np.uint32) for _ in range(2))
    sign = (((src ^ dst) & 7) < 3).astype(np.int8) * -2 + 1
    want = ctx.vertex_counts(src, dst, sign, strategy="hash")
    assert want.sum() > 2_000_000
    np.testing.assert_array_equal(ctx.vertex_counts(src, dst, sign), want)
