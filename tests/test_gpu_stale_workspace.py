"""Nothing that a workspace held before a launch reaches its results: the scratch and the partials
are NaN when the launch under test begins."""
import pytest
import torch

from quantem_b200 import ops
from tests.conftest import rel
from tests.test_gpu_batch_paths import _problem

pytestmark = pytest.mark.gpu


def _poison(device):
    ws = ops.workspace(device)
    for t in (ws.scratch, ws.partials, ws.loss_part):
        if t is not None:
            t.fill_(float("nan"))
    return ws


def _indices(B, invalid):
    """Every position, or with the second and fifth of six replaced by ones that do not exist (whole blocks
    of one or two positions start with, end with and consist of invalid indices)."""
    idx = torch.arange(B, device="cuda")
    if invalid:
        idx[1::6], idx[4::6], idx[-2:] = B, -1, B + 3
    return idx


CASES = [(n, P, kind) for n, P in [(64, 1), (64, 3), (96, 1), (96, 2), (128, 1), (128, 2)]
         for kind in ("plain", "positions", "analytic")] + [(256, 2, "plain")]


@pytest.mark.parametrize("n,P,kind", CASES)
@pytest.mark.parametrize("invalid", [False, True])
def test_poisoned_workspace(cuda_device, n, P, kind, invalid):
    B = 7 if n == 256 else 2 * ops.resident_ctas(n)
    obj, probe, prop, pos, targets = _problem(n, 2, P, B, n + 20, n + 23, seed=P)
    mask, idx = torch.ones((n, n), device="cuda"), _indices(B, invalid)

    def run():
        if kind == "analytic":
            return ops.batch_analytic(obj, probe, prop, pos, idx, targets, mask, B, 100.0)
        g = torch.zeros((B, 2), device="cuda") if kind == "positions" else None
        out = ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, B, 100.0, grad_positions=g)
        return (*out, g) if g is not None else out

    run()  # the workspace has its size
    ws = _poison(obj.device)
    a = [t.clone() for t in run()]
    assert ops.read_status(obj.device)["invalid_indices"] == (2 * int(((idx < 0) | (idx >= B)).sum()))
    ws.scratch.zero_(), ws.partials.zero_(), ws.loss_part.zero_()
    b = run()
    ops.read_status(obj.device)
    for x, y in zip(a, b):  # the object's atomic sums differ in their order: sqrt(B) eps
        assert bool(torch.isfinite(torch.view_as_real(x) if x.is_complex() else x).all())
        assert rel(x.cpu().numpy(), y.cpu().numpy()) < 4e-7 * max(4.0, B ** 0.5)


@pytest.mark.parametrize("n", [64, 96, 128])
def test_block_of_invalid_positions_alone(cuda_device, n):
    """A launch none of whose positions exist: zero gradients, whatever the partials held."""
    obj, probe, prop, pos, targets = _problem(n, 2, 2, 6, n + 20, n + 23)
    mask = torch.ones((n, n), device="cuda")
    idx = torch.full((6,), -1, dtype=torch.int64, device="cuda")
    ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, 6, 100.0, grid=3)
    _poison(obj.device)
    loss, go, gp = ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, 6, 100.0, grid=3)
    ops.read_status(obj.device)
    assert float(loss) == 0.0 and not go.any() and not gp.any()
