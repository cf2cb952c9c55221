"""Arcs counted by one thread where the head side's keys are made: shorter
lists around the limit of 8 entries against longer ones of many lengths, lists
that keep arcs for the tail side beside them, and warps whose arcs span
graphs; totals, per-vertex and per-graph counts against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def fans(k, longs, seed):
    """For every length L of `longs`: two adjacent vertices that share k
    neighbours, one of them with L more neighbours of its own."""
    rng = np.random.default_rng(seed)
    src, dst, at = [], [], 0
    for L in longs:
        u, v = at, at + 1
        shared = np.arange(at + 2, at + 2 + k)
        own = np.arange(at + 2 + k, at + 2 + k + L)
        ring = np.concatenate([shared, own])  # neighbours of some degree, some of them adjacent
        src += [[u], np.full(k, u), np.full(k, v), np.full(L, u), ring[:-1], ring[:-2]]
        dst += [[v], shared, shared, own, ring[1:], ring[2:]]
        at += 2 + k + L
    a, b = np.concatenate(src), np.concatenate(dst)
    p = rng.permutation(at).astype(np.uint32)
    a, b = p[a], p[b]
    lo, hi = np.minimum(a, b).astype(np.int64), np.maximum(a, b).astype(np.int64)
    return a, b, np.where((lo * 7 + hi * 13) % 5 < 2, -1, 1).astype(np.int8)


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 10, 17, 40])
def test_limit(ctx, k):
    g = fans(k, [0, 1, 6, 7, 8, 9, 30, 120, 130, 1100, 4200], k)
    csr = oracle.ForwardCSR(*g)
    for persistent in (False, True):
        assert ctx.count(*g, persistent=persistent).as_tuple() == csr.count()
        np.testing.assert_array_equal(ctx.vertex_counts(*g, persistent=persistent),
                                      csr.vertex_counts())


@pytest.mark.parametrize("G", [3, 90])
def test_graphs_share_warps(ctx, G):
    graphs = [fans(1 + g % 12, [g % 5, 3 * (g % 7)], g) for g in range(G)]
    graphs.insert(G // 2, fans(9, [3000, 5], 77))
    want = [oracle.count_arrays(*x) for x in graphs]
    for persistent in (True, False):
        assert [c.as_tuple() for c in ctx.count_batch(graphs, persistent=persistent)] == want
