"""The column runs that a job starts from: filled by its own blocks up to 65536
rows, by the set-up kernels above; in single calls and in a batch, on wide and
on narrow clusters, equal to the oracle's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matrix(R, nnz, seed):
    """Entries crowded into a few hundred segments over all of the rows, so that groups are invalid."""
    rng = np.random.default_rng(seed)
    c = rng.integers(0, 800, nnz) + (rng.random(nnz) < 0.5) * (R - 800)
    key = np.unique((R * rng.random(nnz) ** 2).astype(np.int64) * R + c)
    return R, (key // R).astype(np.int32), (key % R).astype(np.int32), np.ones(len(key), np.float32)


@pytest.mark.parametrize("R", [65536, 65544, 131072])
@pytest.mark.parametrize("cluster", ["1", "2", "16"])
def test_runs_match_oracle(ctx, monkeypatch, R, cluster):
    mat = _matrix(R, 60000, R)
    monkeypatch.setenv("VNM_NM_CLUSTER", cluster)
    for N, M in ((1, 4), (1, 8)):
        ores, _, _, opos = oracle.nm_run(*mat, N, M, 0)
        assert ores[4] > 3  # rounds
        res, pos = ctx.nm_reorder(*mat, N, M, 0)
        assert np.array_equal(res, ores) and np.array_equal(pos, opos)


@pytest.mark.parametrize("small", [3, 60, 200])
def test_batch_with_a_large_matrix(ctx, small):
    mats = [_matrix(65544, 40000, 7)] + [_matrix(2048 + 8 * b, 4000, b) for b in range(small)]
    res, pos = ctx.nm_reorder_batch(mats, 1, 8, 0)
    for b, m in enumerate(mats):
        r1, p1 = ctx.nm_reorder(*m, 1, 8, 0)
        assert np.array_equal(res[b], r1) and np.array_equal(pos[b], p1), b
