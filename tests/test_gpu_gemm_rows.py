"""The int4 product of many rows, calls one behind the other: every call gives the same bits, and the values of
the general-shape CUDA-core kernel."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(9, 3584, 18944), (32, 3584, 4736), (200, 3584, 18944), (1000, 3584, 4608)])
def test_calls_in_a_row_agree(M, K, N):
    """Enough blocks and weight boxes that a ring slot is refilled while its readers wait for activations."""
    from cpp_tensorlib_b200 import cuda as tl
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = tl.to_q4(torch.randn((K, N), generator=g, device="cuda") * 0.02)
    xs = [torch.randn((M, K), generator=g, device="cuda") for _ in range(2)]
    want = [tl.gemm_q4(x, w, simt=True) for x in xs]
    first = [tl.gemm_q4(x, w) for x in xs]
    rest = [[tl.gemm_q4(x, w) for x in xs] for _ in range(8)]
    for a, b in zip(want, first):
        # f32 sums of K <= 3584 products in another order: about 2^-24 sqrt(K) = 4e-6 of a result, 25 times that for the largest
        assert (a - b).abs().max().item() < 1e-4 * a.std().item()
    for r in rest:
        assert all(torch.equal(a, b) for a, b in zip(first, r))


@pytest.mark.parametrize("M,K,N", [
    (9, 128, 100),        # one tile of half a box: one block
    (32, 384, 129),       # two tiles, the second of one row; a box and a half
    (33, 2048, 256),      # few tiles, every box a block of its own
    (65, 4864, 896),      # tiles of several blocks, ragged on both sides
    (517, 896, 1152),
    (300, 18944, 3584),   # ranges that begin and end inside tiles
    (1000, 3584, 4608),   # whole tiles, two to a block
])
def test_tiles_shared_by_blocks(M, K, N):
    """Parts of a tile are summed in the order of k by whichever block is last: every call gives the same bits.
    With alpha and beta, as the CUDA-core kernel within f32 sums in another order: about 2^-24 sqrt(K) <= 8e-6 of a
    result, 25 times that for the largest."""
    from cpp_tensorlib_b200 import cuda as tl
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    w = tl.to_q4(torch.randn((K, N), generator=g, device="cuda") * 0.02)
    x = torch.randn((M, K), generator=g, device="cuda")
    want = tl.gemm_q4(x, w, alpha=1.5, beta=0.25, simt=True)
    got = [tl.gemm_q4(x, w, alpha=1.5, beta=0.25) for _ in range(6)]
    assert (want - got[0]).abs().max().item() < 2e-4 * want.std().item()
    assert all(torch.equal(got[0], a) for a in got[1:])


@pytest.mark.parametrize("M,K,N", [(8, 18944, 256), (33, 2048, 256), (300, 18944, 3584)])
def test_tickets_are_cleared_with_the_status(M, K, N):
    """Whatever count overlapping products left, the products behind a cleared status are right."""
    from cpp_tensorlib_b200 import check, cuda as tl, lib
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = tl.to_q4(torch.randn((K, N), generator=g, device="cuda") * 0.02)
    x = torch.randn((M, K), generator=g, device="cuda")
    want = tl.gemm_q4(x, w)
    torch.cuda.synchronize()
    for value in (1, 255):
        check(lib().tlb_debug_gemm_tickets(value))
        check(lib().tlb_device_status(None, 1))
        for _ in range(2):
            y = torch.zeros_like(want)
            tl.gemm_q4(x, w, y=y)
            assert torch.equal(want, y)


@pytest.mark.parametrize("M,K,N", [(3, 18944, 3584), (8, 18944, 129), (5, 11008, 500), (8, 3584, 1000)])
def test_few_rows_of_deep_products(M, K, N):
    """Rows whose activations do not fit the skinny kernel's shared memory at once (the last case needs two launches and
    stays there): the CUDA-core kernel's values within f32 sums in another order, about 2^-24 sqrt(K) <= 8e-6 of a result, 25
    times that for the largest; the same bits on every call and in a captured graph."""
    from cpp_tensorlib_b200 import cuda as tl
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    w = tl.to_q4(torch.randn((K, N), generator=g, device="cuda") * 0.02)
    x = torch.randn((M, K), generator=g, device="cuda")
    want = tl.gemm_q4(x, w, simt=True)
    got = tl.gemm_q4(x, w)
    assert (want - got).abs().max().item() < 2e-4 * want.std().item()
    y, graph = torch.zeros_like(got), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tl.gemm_q4(x, w, y=y)
    graph.replay()
    assert torch.equal(got, y) and torch.equal(got, tl.gemm_q4(x, w))


@pytest.mark.parametrize("M,K,N,rows", [(8, 18944, 512, 3000), (32, 3584, 512, 4500), (300, 896, 1152, 6000)])
def test_captured_products_outlive_larger_ones(M, K, N, rows):
    """A product that needs more scratch than any before it, run between two replays of a captured product: the graph
    gives the same bits and leaves memory that was allocated meanwhile alone."""
    from cpp_tensorlib_b200 import cuda as tl
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = tl.to_q4(torch.randn((K, N), generator=g, device="cuda") * 0.02)
    x = torch.randn((M, K), generator=g, device="cuda")
    want = tl.gemm_q4(x, w)
    y, graph = torch.zeros_like(want), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tl.gemm_q4(x, w, y=y)
    graph.replay()
    assert torch.equal(want, y)
    wide = tl.to_q4(torch.zeros((18944, 128), device="cuda"))
    tl.gemm_q4(torch.zeros((rows, 18944), device="cuda"), wide)
    torch.cuda.empty_cache()
    others = [torch.full((1 << n,), 7, dtype=torch.uint8, device="cuda") for n in range(20, 30) for _ in range(2)]
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(want, y)
    assert all(bool((t == 7).all()) for t in others)


FRESH = """
import torch
from cpp_tensorlib_b200 import check, lib, cuda as tl
check(lib().tlb_init(0))
w = tl.to_q4(torch.randn((18944, 512), device="cuda") * 0.02)
x = torch.randn((8, 18944), device="cuda")
y, graph = torch.zeros((8, 512), device="cuda"), torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    tl.gemm_q4(x, w, y=y)
graph.replay()
tl.gemm_q4(torch.randn((64, 18944), device="cuda"), w)
assert torch.equal(y, tl.gemm_q4(x, w))
"""


def test_few_rows_captured_before_any_other_product():
    """Which kernel a product takes follows from its shape: captured as the first product of a process it gives the
    bits of a later call."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", FRESH], cwd=root, check=True, timeout=300)
