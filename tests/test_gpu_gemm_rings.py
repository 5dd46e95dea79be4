"""Products of several rounds (two CTAs to an SM, the short ring) against the same rows in one round (the
deep ring) and against PyTorch."""
import pytest
import torch

from quantem_b200.core.ml import kernels as kk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 16, 30, 32, 40, 64])
@pytest.mark.parametrize("K", [8, 64, 72, 320, 584])
def test_short_ring_matches_deep_ring(cuda_device, N, K):
    """The same products and sums, element by element: equal.  Rows end inside a tile; K covers less than
    one k-block, a whole one, remainders, and more than one turn of both rings."""
    M = 148 * 128 + 77
    g = torch.Generator(device="cuda").manual_seed(N * 1000 + K)
    A = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    B = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    out, parts = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    kk.gemm(A, B, out, bias=bias)
    for r in range(0, M, 8192):
        kk.gemm(A[r:r + 8192], B, parts[r:r + 8192], bias=bias)
    assert torch.equal(out, parts)
    # float32 sums of K exact products: K 2^-24 of the sum of their sizes
    ref = A.double() @ B.double().T + bias.double()
    size = A.double().abs() @ B.double().abs().T + bias.double().abs()
    assert bool(((out.double() - ref).abs() <= (K + 1) * 2.0 ** -24 * size).all())
