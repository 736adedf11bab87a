"""Two host threads, each with its own context, sort rows at once: the launch
shape of one call's rounds (69 to 118 KB of shared memory a block) must not
depend on what the other thread sorts meanwhile.  And the last row count that
one cluster holds, with the first that it does not, against the general path."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _entries(m, nnz, seed):
    rng = np.random.default_rng(seed)
    key = np.unique((m * rng.random(nnz) ** 3).astype(np.int64) * m + (m * rng.random(nnz) ** 3).astype(np.int64))
    return (key // m).astype(np.int32), (key % m).astype(np.int32)


def test_two_threads_sort_at_once():
    import vnm_gb300
    jobs = {40000: 30, 1000: 600}  # rows -> calls, about as long on either thread
    inputs = {m: _entries(m, 8 * m, m) for m in jobs}
    with_one = vnm_gb300.Context(0)
    want = {m: with_one.vnm_reorder(m, m, *inputs[m], 8, 32) for m in jobs}
    with_one.close()
    failed = []

    def work(m):
        ctx = vnm_gb300.Context(0)
        try:
            for _ in range(jobs[m]):
                for a, b in zip(ctx.vnm_reorder(m, m, *inputs[m], 8, 32), want[m]):
                    assert np.array_equal(a, b), m
        except Exception as e:
            failed.append((m, repr(e)))
        ctx.close()

    threads = [threading.Thread(target=work, args=(m,)) for m in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("m", [65536, 65537])
def test_the_largest_cluster(ctx, monkeypatch, m):
    r, c = _entries(m, 4 * m, m)
    new = ctx.vnm_reorder(m, m, r, c, 8, 64)
    monkeypatch.setenv("VNM_VS_ROWS", "0")
    for a, b in zip(new, ctx.vnm_reorder(m, m, r, c, 8, 64)):
        assert np.array_equal(a, b)
