"""The row sort on the original rows (one cluster holds all rows) against the
general path that sorts the entries: block and cluster edges, several rows a
thread, long and equal rows, empty rows, entries in any order, matrices that
are not square, every group size; and against the oracle where it is quick."""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _general(f):
    os.environ["VNM_VS_ROWS"] = "0"
    try:
        return f()
    finally:
        del os.environ["VNM_VS_ROWS"]


def _power_law(m, n, nnz, seed):
    """Distinct positions, hubs first, in random order; a fifth of the rows repeat another row's columns."""
    rng = np.random.default_rng(seed)
    r = (m * rng.random(nnz) ** 3).astype(np.int64)
    c = (n * rng.random(nnz) ** 3).astype(np.int64)
    key = np.unique(r * n + c)
    r, c = key // n, key % n
    src, dst = rng.integers(0, m, m // 5 + 1), rng.integers(0, m, m // 5 + 1)
    copies = []
    for a, b in zip(src[:200], dst[:200]):
        copies.append(b * n + c[r == a])
    key = np.unique(np.concatenate([key] + copies))
    key = key[rng.permutation(len(key))]
    return (key // n).astype(np.int32), (key % n).astype(np.int32)


def _same(ctx, m, n, r, c, M, V):
    new = ctx.vnm_reorder(m, n, r, c, M, V)
    old = _general(lambda: ctx.vnm_reorder(m, n, r, c, M, V))
    for a, b in zip(new, old):
        assert np.array_equal(a, b), (m, n, M, V)
    assert np.array_equal(ctx.vnm_eval(m, n, r, c, M, V), _general(lambda: ctx.vnm_eval(m, n, r, c, M, V)))
    return new


@pytest.mark.parametrize("M", [2, 3, 4, 5, 6, 7, 8])
def test_group_sizes_and_the_oracle(ctx, M):
    m = 40 * M + 3  # padded inside
    r, c = _power_law(m, m, 6 * m, M)
    out, rr, cc, pos = _same(ctx, m, m, r, c, M, 16)
    o5, orr, occ, opos = oracle.vnm_run(m, m, r, c, M, 16)
    assert out.tolist() == o5.tolist() and np.array_equal(pos, opos)
    assert np.array_equal(rr, orr) and np.array_equal(cc, occ)


@pytest.mark.parametrize("m", [1, 31, 1023, 1024, 1025, 2049, 8200, 16384, 16385, 40000])
def test_block_and_cluster_edges(ctx, m):
    r, c = _power_law(m, m, 8 * m, m)
    _same(ctx, m, m, r, c, 8, 32)


@pytest.mark.parametrize("m,n", [(64, 640), (1000, 1504), (4, 9000)])
def test_not_square(ctx, m, n):
    r, c = _power_law(m, min(m, n), 10 * m, n)
    _same(ctx, m, n, r, c, 8, 8)


def test_equal_rows_and_no_entries(ctx):
    m = 2000
    c = np.tile(np.arange(40, dtype=np.int32) * 17, m)  # every row the same 40 entries: 40 levels of one group
    r = np.repeat(np.arange(m, dtype=np.int32), 40)
    _same(ctx, m, m, r, c, 8, 64)
    e = np.zeros(0, np.int32)
    _same(ctx, m, m, e, e, 8, 64)
