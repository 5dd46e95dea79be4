"""The soft object constraints over the forms that pick their kernel: planes that fill their tiles and narrow
ones, few and many slices (runs of slices, their ends), all object types."""
import numpy as np
import pytest
import torch

from oracle import ptycho_oracle as O
from quantem_b200 import ops
from tests.conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 300, 260), (2, 510, 516), (5, 256, 256), (9, 200, 200), (64, 100, 96),
                                   (200, 64, 64), (3, 2000, 36), (8, 70, 64), (1, 8, 32), (2, 2, 2)])
@pytest.mark.parametrize("obj_type", ["complex", "pure_phase", "potential"])
def test_soft_constraints_any_form(cuda_device, shape, obj_type):
    """Against the FP64 oracle: the gradient is made of signs, so an element whose difference rounds to the
    other side is off by a whole step; float32 differences of values of size 1 do that for 2^-24 / 0.1 of the
    elements.  The loss is a mean of absolute differences: a few eps."""
    rng = np.random.default_rng(sum(shape))
    if obj_type == "potential":
        x = rng.uniform(0.0, 1.0, shape).astype(np.float32)
    else:
        x = (rng.uniform(0.5, 1.0, shape) * np.exp(1j * rng.uniform(-1, 1, shape))).astype(np.complex64)
    kw = dict(tv_weight_z=0.3, tv_weight_xy=0.2, surface_zero_weight=0.1)
    t = torch.tensor(x, device=cuda_device, requires_grad=True)
    loss = ops.soft_constraint_loss(t, obj_type, **kw)
    loss.backward()
    want, grad = O.soft_constraint_loss(x.astype(np.float64 if obj_type == "potential" else np.complex128), obj_type, **kw)
    assert abs(float(loss.detach()) - want) < 4e-6 * abs(want)
    g = t.grad.cpu().numpy()
    step = np.abs(grad).max()
    wrong = np.abs(g - grad) > 1e-4 * step
    assert wrong.mean() < 1e-5 + 2.0 / grad.size
    assert rel(np.where(wrong, grad, g), grad) < 1e-5


@pytest.mark.parametrize("S,n", [(200, 128), (64, 200)])
def test_many_slices_use_the_device(cuda_device, S, n):
    """Many slices of a small plane: within a few copies per evaluated value (one block per tile marching all
    slices took 330 us at 200 x 128 x 128 and 209 us for a potential, 12 and 16 times a copy)."""
    def us(f):
        best = float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                f()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 100)
        return best

    for obj_type, most in (("complex", 11), ("potential", 8)):
        x = torch.rand(S, n, n, device="cuda") + 0.5
        x = x if obj_type == "potential" else torch.polar(x, x)
        y, fn = torch.empty_like(x), lambda: ops.soft_constraint_loss(x, obj_type, 0.3, 0.2, 0.0)
        copy = us(lambda: y.copy_(x))
        assert us(fn) < most * max(copy, 10.0) + 15.0
