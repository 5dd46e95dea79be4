"""The Butterworth filter's line transforms at lengths with every radix (2, 3, 4, 5, 8), primes
without a butterfly, one and several of them, length 1, and the longest that fits."""
import numpy as np
import pytest
import torch

from oracle import ptycho_oracle as O
from quantem_b200 import ops
from tests.conftest import rel

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 7), (2, 3), (4, 5), (8, 13), (16, 15), (64, 60), (45, 49), (77, 91), (510, 516), (509, 521),
         (37 * 13, 128), (961, 30), (1024, 1023), (2048, 10), (3, 6144), (6143, 4), (5184, 2)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("real", [False, True])
def test_butterworth_any_size(cuda_device, size, real):
    """Against the FP64 oracle.  A transform of n terms in float32 is off by a few eps sqrt(log2 n)
    relative (butterfly radices) or eps sqrt(p) (a prime p by its sum): 2^-24 (8 + 2 sqrt(p))."""
    rng = np.random.default_rng(size[0] * 10007 + size[1])
    S = 3
    x = 0.7 + 0.2 * rng.standard_normal((S, *size))
    if not real:
        x = x + 0.3j * rng.standard_normal((S, *size))
    dt, ct = (np.float32, np.float64) if real else (np.complex64, np.complex128)
    x = x.astype(dt)
    env = O.butterworth_env(size, (0.2, 0.3), q_lowpass=1.1, q_highpass=0.05)
    t = torch.tensor(x, device=cuda_device)
    e = torch.tensor(env, device=cuda_device)
    y = ops._butter(t, e, vjp=False).cpu().numpy()
    g = ops._butter(t, e, vjp=True).cpu().numpy()

    def largest_prime(n):
        p, d = 1, 2
        while n > 1:
            while n % d == 0:
                n, p = n // d, d
            d += 1
        return p

    tol = 2.0 ** -24 * (8 + 2 * max(largest_prime(size[0]), largest_prime(size[1])) ** 0.5) * 2
    assert rel(y, O.butterworth(x.astype(ct), env.astype(np.float64))) < tol
    assert rel(g, O.butterworth_vjp(x.astype(ct), env.astype(np.float64), real)) < tol
