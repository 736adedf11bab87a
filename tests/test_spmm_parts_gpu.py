"""Tiles of the tensor-core SpMM cut into several parts of their K-steps:
full V:2:M operands of few rows (each V-block row of a tile brings its own
K-steps, so that a smaller V means more parts), ragged last stages, column
counts of each block width, and V-blocks sparse enough for the residual
kernel to have written the tile's rows first."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [16, 64, 128])
@pytest.mark.parametrize("n,dtype", [(64, "bf16"), (128, "fp16"), (192, "bf16"), (256, "fp16"), (320, "bf16")])
def test_split_tiles_match_float64(ctx, V, n, dtype):
    import torch
    import vnm_gb300
    from vnm_gb300 import synth
    R, r, c, v = synth.vnm_structured(1152, 8, V, seed=V)
    # thin out some V-blocks: they become residual entries of the same rows
    rng = np.random.default_rng(n)
    block = (r // V) * (R // 8) + c // 8
    thin = rng.random(block.max() + 1) < 0.1
    keep = ~thin[block] | (rng.random(len(r)) < 0.05)
    r, c, v = r[keep], c[keep], v[keep]
    tdt = torch.bfloat16 if dtype == "bf16" else torch.float16
    B = torch.randn((R, n), generator=torch.Generator().manual_seed(n)).to(tdt)
    A = vnm_gb300.SpmmMatrix(ctx, R, r, c, v, 8, V, dtype)
    info = A.info()
    assert info["residual_nnz"] > 0 and info["tensor_tiles"] == 9 and info["ksteps"] >= 9 * 30
    ref = oracle.spmm_f64(R, r, c, v.astype(np.float64), B.float().numpy().astype(np.float64))
    Bd = B.cuda()
    C = A.run(Bd)
    # values rounded to 16 bits inside their V-block's scale: the SpMM's bound
    assert oracle.rowwise_rel_err(C.cpu().numpy().astype(np.float64), ref) <= 1e-2
    for _ in range(2):  # the same sums in the same order, whichever part ends first
        assert torch.equal(A.run_async(Bd), C)
    A.check()
    A.close()
