"""Scratch of the reorder's calls a row of the matrix: what the header states,
for the cluster size the call runs on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 1 << 22


@pytest.mark.parametrize("call,jobs,blocks", [("pair_score", 1, 1), ("reorder", 1, 8), ("search", 4, 8)])
def test_scratch_bytes_a_row(call, jobs, blocks):
    import torch
    import vnm_gb300
    r = np.arange(3, dtype=np.int32)
    v = np.ones(3, np.float32)
    free = torch.cuda.mem_get_info()[0]
    with vnm_gb300.Context(0) as ctx:
        if call == "pair_score":
            ctx.nm_pair_score(ROWS, r, r, v, 2, 4, 0, 1)
        elif call == "reorder":
            ctx.nm_reorder(ROWS, r, r, v, 2, 4, 0)
        else:
            ctx.nm_search(ROWS, r, r, v, 2, 4)
        used = free - torch.cuda.mem_get_info()[0]
    # the header's bytes a row and the result's 4 a row, a quarter more, and 32 MB for what does not grow with the rows
    assert used <= ROWS * (136 + jobs * (8 * blocks + 28) + 4) * 5 // 4 + (32 << 20), used / ROWS
