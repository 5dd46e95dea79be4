"""Where the forward kernel sums the mode intensities: nowhere (one mode), in shared memory, or in the output
array.  The loss and the intensities are those of the adjoint launch, which sums in its scratch."""
import pytest
import torch

from quantem_b200 import ops
from tests.test_gpu_batch_paths import _problem
from tests.test_gpu_small_launches import device_us

pytestmark = pytest.mark.gpu


def _call(n, S, P, B, seed=0):
    obj, probe, prop, pos, targets = _problem(n, S, P, B, n + 30, n + 41, seed=seed)
    idx, mask, ph = torch.arange(B, device="cuda"), torch.ones((n, n), device="cuda"), ops.fft2(probe)

    def fwd(want):
        return ops.batch_forward(obj, probe, prop, pos, idx, targets, mask, B, 100.0, probe_hat=ph, want_intensity=want)

    def adj():
        return ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, B, 100.0, probe_hat=ph)
    return fwd, adj


@pytest.mark.parametrize("n,S,P", [(64, 1, 1), (64, 2, 3), (64, 40, 2), (96, 2, 1), (96, 3, 2), (128, 2, 1), (128, 2, 4),
                                   (128, 13, 2), (128, 14, 2), (128, 15, 3)])
def test_forward_matches_adjoint_loss(cuda_device, n, S, P):
    """The same products and sums of squares per element; only the order of the double loss sums differs."""
    fwd, adj = _call(n, S, P, 5, seed=S + P)
    a, b, c = fwd(True), fwd(False), adj()
    assert abs(float(a["loss"]) - float(c[0])) <= 2e-7 * abs(float(c[0]))
    assert abs(float(b["loss"]) - float(c[0])) <= 2e-7 * abs(float(c[0]))
    assert bool(torch.isfinite(a["intensity"]).all()) and b["intensity"] is None
    assert torch.equal(a["intensity"], fwd(True)["intensity"])


@pytest.mark.parametrize("n,S,P,B", [(128, 1, 4, 148), (128, 2, 8, 148), (96, 9, 1, 296)])
def test_intensities_cost_their_writing(cuda_device, n, S, P, B):
    """Launches with and without the intensities: summing modes through global memory made the first 13 %
    slower, a tile that a single mode does not need made the second 36 % slower (one resident block less)."""
    fwd, _ = _call(n, S, P, B)
    with_, without = device_us(lambda: fwd(True)), device_us(lambda: fwd(False))
    assert with_ < 1.08 * without + 1.0 and without < 1.08 * with_ + 1.0, (with_, without)
