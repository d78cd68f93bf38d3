"""One to eight rows of int4 products: blocks that own row tiles, and five to eight rows in one pass over the weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [
    (1, 896, 4864), (1, 896, 17), (1, 3584, 4608), (1, 2048, 16),   # blocks own row tiles: several, one, ragged
    (4, 896, 4865), (8, 896, 9728), (7, 1024, 100),
    (8, 3584, 18944), (6, 3712, 333), (5, 4352, 40),                # five to eight rows in one pass
    (1, 4864, 896), (3, 3584, 9000), (8, 256, 48), (1, 128, 4000),  # unit ranges; one unit a tile
])
def test_few_rows(M, K, N):
    """f32 sums of K <= 4864 products in another order: about 2^-24 sqrt(K) = 4e-6 of a result, 25 times that for the
    largest; the same bits on every call and in a graph."""
    from cpp_tensorlib_b200 import cuda as tl
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    w = tl.to_q4(torch.randn((K, N), generator=g, device="cuda") * 0.02)
    x = torch.randn((M, K), generator=g, device="cuda")
    want = tl.gemm_q4(x, w, simt=True)
    got = tl.gemm_q4(x, w)
    assert (want - got).abs().max().item() < 1e-4 * max(want.std().item(), 0.5 * 0.02 * K ** 0.5)
    y, graph = torch.zeros_like(got), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tl.gemm_q4(x, w, y=y)
    graph.replay()
    assert torch.equal(got, y) and torch.equal(got, tl.gemm_q4(x, w))
