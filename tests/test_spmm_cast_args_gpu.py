"""run_cast_async refuses what its kernel would read wrongly: other types, too
few rows, rows that are not contiguous or that overlap, host tensors; and takes
every form that its docstring names."""
import pytest

pytestmark = pytest.mark.gpu


def test_cast_product_refuses_other_inputs(ctx):
    import torch
    import vnm_gb300
    from vnm_gb300 import synth
    n, r, c, v = synth.chung_lu(512, 2.1, 8.0, 3)
    A = vnm_gb300.SpmmMatrix(ctx, n, r, c, v, 8, 128, "bf16")
    X = torch.randn((n, 100), generator=torch.Generator().manual_seed(1))
    refused = [X,  # on the host
               X.double().cuda(), X.int().cuda(), X.bool().cuda(), X.cfloat().cuda(),
               X[:-1].cuda(), torch.cat([X, X]).cuda(), X[0].cuda(), X[:, :0].cuda(), X[None].cuda(),
               X.t().contiguous().cuda().t(), torch.cat([X, X], 1).cuda()[:, ::2],
               X[:1].cuda().expand(n, 100), X.reshape(-1).cuda().as_strided((n, 100), (99, 1))]
    for x in refused:
        with pytest.raises(ValueError):
            A.run_cast_async(x)
    want = A.run_cast_async(X.cuda())
    for x in (torch.cat([X, X], 1).cuda()[:, :100], X.cuda().bfloat16()):
        assert torch.equal(A.run_cast_async(x), want)
    L, B, C = vnm_gb300.lib(), torch.empty((n, 128), dtype=torch.bfloat16, device="cuda"), torch.empty((n, 128)).cuda()
    args = [ctx.h, A.h, X.cuda().data_ptr(), 2, 100, 100, B.data_ptr(), 128, C.data_ptr(), 0]
    for at, bad in ((2, args[2] + 2), (3, 3), (4, 99), (6, args[6] + 8), (7, 64), (8, None), (8, args[8] + 8)):
        assert L.vnm_spmm_run_cast_async(*(args[:at] + [bad] + args[at + 1:])) == 1, at  # VNM_ERR_ARG
    A.check()
    A.close()
