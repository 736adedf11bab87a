"""One launch holds all column blocks of a product (256, then 128 and 64
columns): every multiple of 64 up to three blocks, on a residual operand with
split rows and on one with tensor-core tiles of both kinds, against FP64; and
no more launches than at 256 columns."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["residual", "tensor"])
@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
def test_every_column_count_in_one_launch(ctx, kind, dtype):
    import torch
    import vnm_gb300
    from vnm_gb300 import synth
    if kind == "residual":
        R, r, c, v = synth.chung_lu(3000, 2.1, 20.0, 5)
        new = np.random.default_rng(1).permutation(R).astype(np.int32)  # no dense corner
        r, c = new[r], new[c]
        A = vnm_gb300.SpmmMatrix(ctx, R, r, c, v, 8, 128, dtype)
        assert A.info()["tensor_tiles"] == 0 and A.info()["split_chunks"] > 0
    else:
        R, r, c, v = synth.vnm_structured(640, 8, 32, seed=6)
        A = vnm_gb300.SpmmMatrix(ctx, R, r, c, v, 8, 32, dtype)
        assert A.info()["tensor_tiles"] == 5
    g = torch.Generator().manual_seed(7)
    X = torch.randn((R, 704), generator=g).to(torch.bfloat16 if dtype == "bf16" else torch.float16)
    ref = oracle.spmm_f64(R, r, c, v.astype(np.float64), X.float().numpy().astype(np.float64))
    launches = {}
    for n in range(64, 705, 64):
        C = A.run_async(X[:, :n].contiguous().cuda())
        launches[n] = ctx.last_launch_count
        # values rounded to 16 bits inside their V-block's scale: the SpMM's bound
        assert oracle.rowwise_rel_err(C.cpu().numpy().astype(np.float64), ref[:, :n]) <= 1e-2, n
    A.check()
    assert set(launches.values()) == {launches[256]}, launches
    A.close()
