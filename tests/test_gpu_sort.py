"""The radix sort behind every CSR at the edges of its tiles and of its three
tile sizes (1,024, 2,048 and 4,096 keys), through the CSR it builds: the
forward CSR equals the oracle's, whose lists are sorted on the host."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def edges(m, seed):
    rng = np.random.default_rng(seed)
    n = max(4, m // 3)
    src = rng.integers(0, n, m).astype(np.uint32)
    dst = ((src + 1 + rng.integers(0, n - 1, m)) % n).astype(np.uint32)
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    return src, dst, np.where((lo * 7 + hi * 13) % 3 == 0, -1, 1).astype(np.int8)


@pytest.mark.parametrize("m", [1, 2, 31, 1023, 1024, 1025, 2049, 4097, 606_207, 606_208, 606_209,
                               607_233, 2_424_831, 2_424_832, 2_424_833, 2_428_930])
def test_sort_tile_edges(ctx, m):
    src, dst, sign = edges(m, m)
    got = ctx.build_forward_csr(src, dst, sign)
    want = oracle.ForwardCSR(src, dst, sign).arrays()
    assert (got.n, got.m) == (want["n"], want["m"])
    for k in ("offsets", "edges", "signs", "fdeg", "rank"):
        np.testing.assert_array_equal(getattr(got, k), want[k], err_msg=k)


def test_skewed_digits(ctx):
    # One hub: all arcs share their head, so a digit holds every key of a tile.
    n = 700_001
    src = np.arange(1, n, dtype=np.uint32)
    dst = np.zeros(n - 1, np.uint32)
    sign = np.where(src % 3 == 0, -1, 1).astype(np.int8)
    got = ctx.build_forward_csr(src, dst, sign)
    want = oracle.ForwardCSR(src, dst, sign).arrays()
    for k in ("offsets", "edges", "signs", "fdeg", "rank"):
        np.testing.assert_array_equal(getattr(got, k), want[k], err_msg=k)
