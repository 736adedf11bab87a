"""The learned search's rounds at the edges of its kernels: segment counts
around the tile of the active list, columns around a chunk of rows.  The
totals are integers and must be those of the permuted matrix."""
import numpy as np
import pytest

import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nseg,M,hub", [(2, 8, 3), (3, 2, 5), (33, 8, 255), (70, 4, 256), (100, 3, 257),
                                        (4095, 2, 513), (4096, 2, 300), (4097, 2, 1), (8200, 8, 4000)])
def test_round_totals_match(ctx, nseg, M, hub):
    import vnm_gb300
    n = nseg * M
    rng = np.random.default_rng(nseg)
    hubs = rng.choice(n, 3, replace=False)
    r = np.concatenate([rng.integers(0, n, 6 * n)] + [rng.choice(n, min(hub, n), replace=False) for _ in hubs])
    c = np.concatenate([rng.integers(0, n, 6 * n)] + [np.full(min(hub, n), h) for h in hubs])
    key = np.unique(r * n + c)
    r, c = (key // n).astype(np.int32), (key % n).astype(np.int32)
    v = np.ones(len(r), np.float32)
    N = max(1, M // 4)
    for objective in (0, 1):
        res, pos, _ = vnm_gb300.nm_learned(ctx, n, r, c, v, N, M, mode=2, objective=objective, targets=4,
                                           max_rounds=4, patience=4, seed=3)
        assert np.array_equal(np.sort(pos), np.arange(n))
        assert mo.nm_totals(n, r, c, v, N, M) == (res["init_invalid"], res["init_retained"])
        after = mo.nm_totals(n, pos[r], pos[c], v, N, M)
        assert after == (res["final_invalid"], res["final_retained"])
        gain = after[1] - res["init_retained"] if objective else res["init_invalid"] - after[0]
        assert gain == res["gain"] >= 0
