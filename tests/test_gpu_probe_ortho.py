"""Cluster orthogonalisation: element counts that leave ragged or empty slices, and windows whose
modes, gradients or running vector do not fit in shared memory."""
import numpy as np
import pytest
import torch

from oracle import ptycho_oracle as O
from quantem_b200.diffractive_imaging.ptycho_utils import orthogonalize_probes
from tests.conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,shape", [(1, (1, 1)), (3, (3, 5)), (2, (65, 67)), (16, (32, 32)), (9, (128, 128)),
                                     (16, (128, 128)), (6, (256, 256)), (2, (512, 512)), (2, (700, 701))])
def test_orthogonalisation_slices_and_placements(cuda_device, P, shape):
    rng = np.random.default_rng(P * 7 + shape[0])
    probe = rng.standard_normal((P, *shape)) + 1j * rng.standard_normal((P, *shape))
    probe = (probe * rng.uniform(0.5, 2.0, (P, 1, 1))).astype(np.complex64).astype(np.complex128)
    g = rng.standard_normal((P, *shape)) + 1j * rng.standard_normal((P, *shape))
    if P > shape[0] * shape[1]:
        pytest.skip("more modes than elements")
    out_o, _, cache = O.gram_schmidt(probe)
    g_o = O.gram_schmidt_vjp(cache, g)
    pt = torch.tensor(probe, dtype=torch.complex64, device=cuda_device, requires_grad=True)
    out = orthogonalize_probes(pt)
    torch.sum(torch.real(torch.conj(torch.tensor(g, dtype=torch.complex64, device=cuda_device)) * out)).backward()
    # P projections of float32 elements with float64 sums: a few eps per projection
    assert rel(out.detach().cpu().numpy(), out_o) < 2e-6
    assert rel(pt.grad.cpu().numpy(), g_o) < 4e-6 * max(1, P / 4)
