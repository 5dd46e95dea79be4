"""MN-major operands of the BF16 GEMM and its narrow tiles, against the K-major product."""
import pytest
import torch

from quantem_b200.core.ml import kernels as kk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,splits", [(1, 8, 8, 1), (36, 288, 16384, 4), (128, 64, 64, 1), (130, 200, 70, 1),
                                          (512, 1152, 16, 1), (32, 9216, 256, 1), (16, 1024, 9216, 1),
                                          (1000, 72, 33, 1), (64, 4608, 130, 2)])
@pytest.mark.parametrize("a_mn", [False, True])
def test_mn_major_operands_match_k_major(cuda_device, M, N, K, splits, a_mn):
    """The same products in the same order: equal bits without split-K, the atomics' order of
    FP32 additions with it (splits - 1 roundings of the result's size)."""
    g = torch.Generator(device=cuda_device).manual_seed(M + N + K)

    def pad(r, c):  # rows on 16-byte boundaries
        return torch.randn((r, (c + 7) // 8 * 8), generator=g, device=cuda_device).to(torch.bfloat16)[:, :c]

    A, B = pad(M, K), pad(K, N)
    Am = A
    if a_mn:
        Am = torch.zeros((K, (M + 7) // 8 * 8), dtype=torch.bfloat16, device=cuda_device)[:, :M]
        Am.copy_(A.T)
    Bk = torch.zeros((N, (K + 7) // 8 * 8), dtype=torch.bfloat16, device=cuda_device)[:, :K]
    Bk.copy_(B.T)
    st = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    want, got = torch.empty((M, N), device=cuda_device), torch.empty((M, N), device=cuda_device)
    kk.gemm(A, Bk, want, status=st)
    kk.gemm_mn(Am, B, got, a_mn, splits=splits, status=st)
    assert int(st) == 0
    if splits == 1:
        assert torch.equal(got, want)
    else:
        assert (got - want).abs().max() <= 8 * splits * 2.0 ** -24 * (A.float().abs() @ B.float().abs()).max()
    exact = A.double() @ B.double()
    assert (want - exact).abs().max() <= 2.0 ** -22 * K ** 0.5 * (A.double().abs() @ B.double().abs()).max()
