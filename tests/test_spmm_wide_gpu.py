"""Products of more columns than a grid's y dimension has blocks for, where
partial rows and partial tiles are added (8 columns of a tile, 64 of a row a
block): the first and the last columns are those of narrow products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("tiles", 65536 * 8 + 64), ("rows", 65536 * 64 + 64)])
def test_more_columns_than_blocks_in_y(ctx, kind, n):
    import torch
    import vnm_gb300
    rng = np.random.default_rng(2)
    if kind == "tiles":  # 48 K-steps a tile: two parts
        R, M = 384, 2
        r, c = (x.reshape(-1).astype(np.int32) for x in np.meshgrid(np.arange(R), np.arange(R), indexing="ij"))
    else:  # one row of two chunks
        R, M = 304, 8
        r, c = np.zeros(300, np.int32), np.arange(300, dtype=np.int32)
    A = vnm_gb300.SpmmMatrix(ctx, R, r, c, rng.standard_normal(len(r)).astype(np.float32), M, 128, "bf16")
    info = A.info()
    assert (info["tensor_tiles"], info["ksteps"], info["split_chunks"]) == ((3, 144, 0) if kind == "tiles" else (0, 0, 2))
    g = torch.Generator(device="cuda").manual_seed(3)
    B = torch.empty((R, n), dtype=torch.bfloat16, device="cuda")
    B[:, :256] = torch.randn((R, 256), generator=g, device="cuda")
    B[:, 256:-64] = 0
    B[:, -64:] = torch.randn((R, 64), generator=g, device="cuda")
    C = A.run_async(B)
    A.check()
    for cols in (slice(0, 256), slice(n - 64, n)):  # blocks of the same width: the same sums
        assert torch.equal(C[:, cols], A.run_async(B[:, cols].contiguous()))
    assert C[:, 256:-64].count_nonzero() == 0
    torch.cuda.synchronize()
    A.close()
    del B, C
    torch.cuda.empty_cache()
