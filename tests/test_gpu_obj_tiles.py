"""Tiled blur and soft-constraint kernels at sizes that cut their tiles (32 x 32 and 32 x 8), with
halos of every kind: none, a few taps, the widest tile halo, and one tap pair beyond it."""
import numpy as np
import pytest
import torch

from oracle import ptycho_oracle as O
from quantem_b200 import ops
from tests.conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 31, 33), (1, 32, 32), (3, 5, 100), (2, 65, 64)])
@pytest.mark.parametrize("ntaps", [1, 3, 7, 33, 35])
@pytest.mark.parametrize("real", [False, True])
def test_blur_tiles(cuda_device, shape, ntaps, real):
    """ntaps products per axis in float32: 2 ntaps eps of the sum of magnitudes (taps sum to 1)."""
    rng = np.random.default_rng(ntaps + shape[1])
    x = rng.standard_normal(shape) + (0 if real else 1j * rng.standard_normal(shape))
    x = x.astype(np.float32 if real else np.complex64)
    taps = rng.uniform(0.1, 1.0, ntaps).astype(np.float32)
    taps = ((taps + taps[::-1]) / (2 * taps.sum())).astype(np.float32)
    got = ops._blur(torch.tensor(x, device=cuda_device), torch.tensor(taps, device=cuda_device)).cpu().numpy()
    want = O.blur(x.astype(np.float64 if real else np.complex128), taps)
    assert np.abs(got - want).max() <= 4 * ntaps * 2.0 ** -24 * np.abs(x).max() * 1.5


@pytest.mark.parametrize("shape", [(1, 2, 2), (2, 9, 31), (3, 8, 32), (5, 17, 65), (3, 100, 7)])
@pytest.mark.parametrize("kind", ["complex", "pure_phase", "potential"])
@pytest.mark.parametrize("weights", [(0.3, 0.2, 0.0), (0.0, 0.5, 0.4), (0.7, 0.0, 0.1)])
def test_soft_loss_tiles(cuda_device, shape, kind, weights):
    """Loss to the rounding of its float32 terms (2^-22 relative), gradient to a few eps."""
    rng = np.random.default_rng(shape[1])
    x = rng.uniform(0.1, 0.9, shape)
    if kind != "potential":
        x = rng.uniform(0.5, 1.2, shape) * np.exp(1j * rng.uniform(-1.5, 1.5, shape))
    x = x.astype(np.float32 if kind == "potential" else np.complex64)
    loss_o, grad_o = O.soft_constraint_loss(x.astype(np.float64 if kind == "potential" else np.complex128), kind, *weights)
    t = torch.tensor(x, device=cuda_device, requires_grad=True)
    loss = ops.soft_constraint_loss(t, kind, *weights)
    loss.backward()
    assert abs(float(loss.detach()) - loss_o) <= 1e-6 * max(abs(loss_o), 1e-3)
    if np.abs(grad_o).max() > 0:
        assert rel(t.grad.cpu().numpy(), grad_o) < 2e-6
