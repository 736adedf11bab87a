"""Where the round kernel keeps its records (a slot a row below a block's
share of 4352 rows, a hashed table above), how the blocks' scores come
together (two to a word, singly for columns of more than 4095 entries in a
block) and which clusters a batch runs on: integers throughout, equal to the
oracle's at the sizes where one way ends and the next begins."""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matrix(R, nnz, seed, hubs=()):
    rng = np.random.default_rng(seed)
    rs, cs = [rng.integers(0, R, nnz)], [rng.integers(0, R, nnz)]
    for col, rows in hubs:
        rs.append(np.arange(rows))
        cs.append(np.full(rows, col))
    key = np.unique(np.concatenate(rs) * R + np.concatenate(cs))
    r, c = (key // R).astype(np.int32), (key % R).astype(np.int32)
    return R, r, c, np.ones(len(r), np.float32)


def _check(ctx, mat, N, M, sched, cs):
    old = os.environ.get("VNM_NM_CLUSTER")
    try:
        os.environ["VNM_NM_CLUSTER"] = str(cs)
        res, pos = ctx.nm_reorder(*mat, N, M, sched)
    finally:
        os.environ.pop("VNM_NM_CLUSTER") if old is None else os.environ.update(VNM_NM_CLUSTER=old)
    ores, _, _, opos = oracle.nm_run(*mat, N, M, sched)
    assert np.array_equal(res, ores) and np.array_equal(pos, opos)


# rows a multiple of M; 16 * 272 = 4352 rows are the most that one block owns directly
@pytest.mark.parametrize("M,R,cs", [(8, 8, 1), (8, 16, 8), (4, 36, 2), (8, 264, 16), (4, 4352, 1), (4, 4356, 1),
                                    (8, 4352, 1), (8, 4368, 1), (2, 8704, 2), (7, 8708, 2), (8, 8704, 2),
                                    (8, 8720, 2), (5, 1000, 4)])
def test_record_places_match_oracle(ctx, M, R, cs):
    mat = _matrix(R, 6 * R, R + M)
    for sched in (0, 3):
        _check(ctx, mat, max(1, M // 4), M, sched, cs)


# a hub column's rows over the two blocks of a cluster, about half each: 4095 a block is the most that packs
@pytest.mark.parametrize("M", [4, 8])
@pytest.mark.parametrize("R,rows", [(8704, 8190), (8704, 8704), (8720, 8720)])
def test_long_columns_match_oracle(ctx, M, R, rows):
    hubs = [(q, rows) for q in (0, 1, 2, 3, M, M + 1, M + 2, 2 * M + 1)]
    _check(ctx, _matrix(R, 3 * R, rows + M, hubs), 2, M, 0, 2)


# the batch sizes at which all jobs run at once on clusters of 8, 4 and 2, and past them
@pytest.mark.parametrize("nmat", [1, 15, 19, 20, 38, 39])
def test_batch_clusters_match_single_runs(ctx, nmat):
    rng = np.random.default_rng(nmat)
    mats = [_matrix(8 * int(rng.integers(1, 60)), int(rng.integers(1, 3000)), 100 * nmat + b) for b in range(nmat)]
    res, pos = ctx.nm_reorder_batch(mats, 2, 8, 1)
    for b, m in enumerate(mats):
        r1, p1 = ctx.nm_reorder(*m, 2, 8, 1)
        assert np.array_equal(res[b], r1) and np.array_equal(pos[b], p1), b


# batches that run their largest jobs on wider clusters beside the others: few, the most (18), more
@pytest.mark.parametrize("large", [1, 6, 18, 20])
def test_batch_wide_jobs_match_single_runs(ctx, large):
    rng = np.random.default_rng(large)
    sizes = [(8 * int(rng.integers(200, 400)), 30000 + 500 * b) for b in range(large)]
    sizes += [(8 * int(rng.integers(1, 60)), int(rng.integers(1, 3000))) for _ in range(160)]
    mats = [_matrix(*sizes[b], 1000 * large + int(b)) for b in rng.permutation(len(sizes))]
    res, pos = ctx.nm_reorder_batch(mats, 2, 8, 0)
    for b, m in enumerate(mats):
        r1, p1 = ctx.nm_reorder(*m, 2, 8, 0)
        assert np.array_equal(res[b], r1) and np.array_equal(pos[b], p1), b
