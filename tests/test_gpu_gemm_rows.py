"""The int4 product of many rows, calls one behind the other: every call gives the same bits, and the values of
the general-shape CUDA-core kernel."""
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
