"""The compressor on entries in row order (no sort by block) and in other
orders, and the radix sort below and above the count at which a pass takes
its offsets from a scan (128 tiles of 4096 keys): values and features are
small integers and powers of two, so every product is exact and the orders
must give the same bits."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nnz", [1, 31, 4095, 4096, 4097, 524287, 524288, 524289, 600001])
@pytest.mark.parametrize("M,V", [(8, 64), (4, 16)])
def test_entry_orders_give_the_same_product(ctx, nnz, M, V):
    import torch
    import vnm_gb300
    R = 4096
    rng = np.random.default_rng(nnz + M)
    key = np.sort(rng.choice(R * R // 8, nnz, replace=False))  # the first rows: dense and sparse blocks
    r, c = (key // (R // 4)).astype(np.int32), (key % (R // 4)).astype(np.int32)
    v = rng.choice(np.array([-2, -1, 1, 2], np.float32), nnz)
    B = torch.from_numpy(rng.integers(-2, 3, (R, 64)).astype(np.float32)).to(torch.bfloat16)
    ref = oracle.spmm_f64(R, r, c, v.astype(np.float64), B.float().numpy().astype(np.float64))
    for order in (np.arange(nnz), np.lexsort((r, c)), rng.permutation(nnz)):
        A = vnm_gb300.SpmmMatrix(ctx, R, r[order], c[order], v[order], M, V, "bf16")
        C = A.run(B.cuda()).cpu().numpy()
        A.close()
        assert np.array_equal(C.astype(np.float64), ref)
