"""The storage of a freed operand goes to the context's next compression only
when the products that were enqueued asynchronously with it have ended."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["residual", "tensor", "graph"])
def test_compression_after_a_free_under_a_running_product(kind):
    import torch
    import vnm_gb300
    from vnm_gb300 import synth
    if kind == "residual":
        nr, r, c, v = synth.rmat(12, 40000, seed=3)  # rows in several chunks among them: partial sums too
        M, V = 4, 64
    else:
        nr, r, c, v = synth.vnm_structured(2048, 8, 128, seed=4)
        M, V = 8, 128
    ctx = vnm_gb300.Context(0)
    B = torch.randn((nr, 128), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    A = vnm_gb300.SpmmMatrix(ctx, nr, r, c, v, M, V, "bf16")
    want = A.run(B)
    C, out = torch.empty_like(want), torch.empty_like(want)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    if kind == "graph":
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            A.run_async(B, C, stream=side)
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)  # some 50 ms: the product still waits when the operand is freed
        if kind == "graph":
            graph.replay()
        else:
            A.run_async(B, C, stream=side)
    A.close()
    other = vnm_gb300.SpmmMatrix(ctx, nr, r, c, 3.0 * v, M, V, "bf16")  # the same sizes: the freed storage fits
    other.run(B, out)
    torch.cuda.synchronize()
    assert torch.equal(C, want)
    assert torch.equal(out, other.run(B))  # nothing of the first product's reached the new operand
    other.close()
    ctx.close()
