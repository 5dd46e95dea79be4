"""The constant that the Butterworth filter takes off a slice stands for its mean, wherever the
slice's values lie: border columns or rows unlike the rest must not set it."""
import numpy as np
import pytest
import torch

from oracle import ptycho_oracle as O
from quantem_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(512, 512), (256, 640), (1024, 256), (510, 516)])
@pytest.mark.parametrize("edge", ["column", "row"])
@pytest.mark.parametrize("real", [False, True])
def test_butterworth_with_an_edge_unlike_the_rest(cuda_device, size, edge, real):
    """A slice near 0 whose first column (or row) is 1: its deviation from its mean is 1/16 to 1/32
    of the edge's value, and the transforms' rounding is relative to that deviation: a few eps for the
    butterfly radices, eps sqrt(p) for a prime p by its sum (43 in 516), and the last addition's own."""
    rng = np.random.default_rng(size[0] + size[1])
    x = 1e-3 * rng.standard_normal((2, *size))
    if not real:
        x = x + 1e-3j * rng.standard_normal((2, *size))
    if edge == "column":
        x[:, :, 0] = 1.0
    else:
        x[:, 0] = 1.0
    dt, ct = (np.float32, np.float64) if real else (np.complex64, np.complex128)
    x = x.astype(dt)
    env = O.butterworth_env(size, (0.2, 0.3), q_lowpass=1.1, q_highpass=0.05)
    t, e = torch.tensor(x, device=cuda_device), torch.tensor(env, device=cuda_device)
    prime = 43 if 516 in size else 1
    dev = np.sqrt(np.mean(np.abs(x - x.mean(axis=(1, 2), keepdims=True)) ** 2))
    for vjp in (False, True):
        y = ops._butter(t, e, vjp=vjp).cpu().numpy()
        want = (O.butterworth_vjp(x.astype(ct), env.astype(np.float64), real) if vjp else
                O.butterworth(x.astype(ct), env.astype(np.float64)))
        err = np.sqrt(np.mean(np.abs(y - want) ** 2))
        assert err < 2.0 ** -24 * ((8 + 2 * prime ** 0.5) * dev + np.sqrt(np.mean(np.abs(want) ** 2)))
