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


@pytest.mark.parametrize("F", [1, 7, 64, 100, 130])
@pytest.mark.parametrize("xdtype,dtype", [("float32", "bf16"), ("float32", "fp16"), ("bfloat16", "fp16"),
                                          ("float16", "fp16")])
def test_cast_product_matches_torch_rounding(ctx, F, xdtype, dtype):
    """Features rounded and padded by the library give bit for bit the product
    of the features rounded and padded by torch, whatever their stride and
    alignment, infinities and overflowing values among them."""
    import torch
    import vnm_gb300
    from vnm_gb300 import gcn, synth
    n, r, c, v = synth.chung_lu(1000, 2.1, 8.0, 3)
    A = vnm_gb300.SpmmMatrix(ctx, n, r, c, v, 8, 128, dtype)
    g = torch.Generator().manual_seed(F)
    X = (100 * torch.randn((n, F), generator=g)).to(getattr(torch, xdtype))
    X[5, 0], X[6, F - 1], X[7, 0] = float("inf"), 70000.0, float("-inf")
    X = X.cuda()
    wide = torch.zeros((n, F + 3), dtype=X.dtype, device="cuda")
    wide[:, 3:] = X
    Xp, _ = gcn._pad_cols(X.to(torch.bfloat16 if dtype == "bf16" else torch.float16))
    want = A.run_async(Xp)[:, :F]
    for x in (X, wide[:, 3:]):
        assert torch.equal(torch.nan_to_num(A.run_cast_async(x), nan=1.25), torch.nan_to_num(want, nan=1.25))
    A.close()
