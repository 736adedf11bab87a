"""A wait of the walk that runs out between two swaps of a round: the job
fails with VNM_ERR_INTERNAL, the recount that still follows looks up columns
of the round only (swaps after the failed one may move a column twice), and
the context keeps working.  The heaps publish nothing (a test hook), so the
walk fails at the first pair whose best swap is tied; many invalid segments
and few distinct gains make that happen after swaps of the same round."""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", ["1", "8"])
@pytest.mark.parametrize("N,M", [(1, 2), (1, 3), (2, 4), (1, 4), (2, 5), (2, 7), (2, 8)])
def test_walk_that_stops_between_swaps(ctx, monkeypatch, N, M, cluster):
    import vnm_gb300
    nr = 40 * M
    rng = np.random.default_rng(100 * M + N)
    key = np.sort(rng.choice(nr * nr, nr * nr // 6, replace=False))
    r, c = (key // nr).astype(np.int32), (key % nr).astype(np.int32)
    v = np.ones(len(key), np.float32)
    monkeypatch.setenv("VNM_NM_CLUSTER", cluster)
    for sched in range(4):
        ores, _, _, opos = oracle.nm_run(nr, r, c, v, N, M, sched)
        with monkeypatch.context() as m:
            m.setenv("VNM_NM_TEST_HOLD_HEAPS", "1")
            m.setenv("VNM_NM_TEST_WAIT_LIMIT", "256")
            with pytest.raises(vnm_gb300.VnmError) as e:
                ctx.nm_reorder(nr, r, c, v, N, M, sched)
            assert e.value.status == 6  # VNM_ERR_INTERNAL
        res, pos = ctx.nm_reorder(nr, r, c, v, N, M, sched)
        assert np.array_equal(res, ores) and np.array_equal(pos, opos)
