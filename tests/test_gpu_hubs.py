"""Hubs in random order: their additions do not serialise in a batch or in a
list of half a million edges (the degree stage of a shuffled star against that
of a list without a hub, device times), and batches with hubs, on both sides of
the sizes from where the hub table is used, count as the oracle does."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def graph(n, m, share, seed):
    """`share` of the edges meet one of three hubs."""
    rng = np.random.default_rng(seed)
    a = rng.integers(0, n, m)
    b = (a + 1 + rng.integers(0, 40, m)) % n
    b = np.where(rng.random(m) < share, rng.integers(0, 3, m) * (n // 3), b)
    swap = rng.random(m) < 0.5
    src, dst = np.where(swap, a, b).astype(np.uint32), np.where(swap, b, a).astype(np.uint32)
    return src, dst, np.where((a * 7 + b * 13) % 3 == 0, -1, 1).astype(np.int8)


def star(n, m, seed):
    src, dst, sign = graph(n, m, 0.0, seed)
    rng = np.random.default_rng(seed + 1)
    hub_is_src = rng.random(m) < 0.5
    src[hub_is_src], dst[~hub_is_src] = 0, 0
    return src, dst, sign


def degree_ms(ctx, call):
    for _ in range(4):
        call()
    times = []
    for _ in range(9):
        call()
        times.append(ctx.last_stats().ms_dedup)
    return sorted(times)[4]


def test_star_in_a_batch(ctx):
    n = m = 4_000_000
    rest = graph(100_000, 400_000, 0.0, 5)
    spread = degree_ms(ctx, lambda b=[graph(n, m, 0.0, 6), rest]: ctx.count_batch(b))
    hub = degree_ms(ctx, lambda b=[star(n, m, 6), rest]: ctx.count_batch(b))
    assert hub < 2.5 * spread, (hub, spread)


def test_star_alone(ctx):
    n = m = 1_000_000
    spread = degree_ms(ctx, lambda g=graph(n, m, 0.0, 7): ctx.count(*g))
    hub = degree_ms(ctx, lambda g=star(n, m, 7): ctx.count(*g))
    assert hub < 2.5 * spread, (hub, spread)


@pytest.mark.parametrize("m", [(1 << 19) - 1, 1 << 19, (1 << 19) + 7, 2_000_003])
def test_counts_with_hubs(ctx, m):
    one = graph(m // 5, m, 0.4, m)
    want = oracle.count_arrays(*one)
    assert sum(want) > 0 and ctx.count(*one).as_tuple() == want
    a = m // 3  # three graphs with m edges in all
    batch = [graph(a // 4, a, 0.5, 1), graph(50, m - a - 100, 0.3, 2), graph(30, 100, 0.9, 3)]
    want = [oracle.count_arrays(*g) for g in batch]
    for persistent in (True, True, True, False):
        assert [c.as_tuple() for c in ctx.count_batch(batch, persistent=persistent)] == want
