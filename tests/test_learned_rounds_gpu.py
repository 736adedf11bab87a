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


def _one_invalid_segment(nseg, N, M, seed):
    # segment 0 holds groups of up to M bits, the others of up to N, with columns of uneven lengths
    rng = np.random.default_rng(seed)
    n = nseg * M
    r, c = [], []
    for i in range(n):
        for s in range(nseg):
            most = M if s == 0 else N
            for k in rng.choice(M, int(rng.integers(0, most + 1)), replace=False):
                if s == 0 or rng.random() < (k + 1.0) / M:
                    r.append(i)
                    c.append(s * M + int(k))
    key = np.unique(np.array(r) * n + np.array(c))
    return n, (key // n).astype(np.int32), (key % n).astype(np.int32), np.ones(len(key), np.float32)


@pytest.mark.parametrize("M,targets", [(2, 1), (2, 512), (3, 15), (3, 227), (4, 9), (4, 128), (5, 6), (5, 81), (6, 4),
                                       (6, 56), (7, 3), (7, 41), (8, 1), (8, 3), (8, 32)])
def test_network_proposes_its_best_candidate(ctx, M, targets):
    """A network whose score is one of the features proposes a candidate with
    the largest such feature of all that exhaustive scoring lists, for each
    feature (scores are BF16 features exactly: no tolerance)."""
    import vnm_gb300
    N = max(1, M // 2)
    mat = _one_invalid_segment(7, N, M, M)
    kw = dict(max_rounds=1, targets=targets, seed=11, dump_every=1, dump_cap=2048)
    _, _, (cands, _) = vnm_gb300.nm_learned(ctx, *mat, N, M, mode=vnm_gb300.LEARNED_EXHAUSTIVE, **kw)
    assert len(cands) == targets * M * M
    net = vnm_gb300.Mlp(ctx, 0)
    for k in range(mo.F):
        w = np.zeros_like(net.get())
        w[k] = w[mo.OFF_W2] = w[mo.OFF_W3] = 1.0  # the first hidden units pass feature k on
        net.set(w)
        _, _, (best, _) = vnm_gb300.nm_learned(ctx, *mat, N, M, mode=vnm_gb300.LEARNED_MLP, net=net, topk=1, **kw)
        assert len(best) == 1
        assert mo.bf16(best[0, k]) == mo.bf16(cands[:, k].max()), k
