"""Branches of the batch kernels that a launch picks by its sizes: windows inside the object's
columns (compile-time offsets) against windows that touch or wrap around an edge, separable
propagators from shared memory against the L1 cache, more CTAs than one per SM."""
import numpy as np
import pytest
import torch

from quantem_b200 import ops
from tests.conftest import rel

pytestmark = pytest.mark.gpu


def _problem(n, S, P, B, ho, wo, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd(*s):
        return torch.randn(s, generator=g, device="cuda")

    obj = torch.polar(1 - 0.2 * torch.rand((S, ho, wo), generator=g, device="cuda"), 0.3 * rnd(S, ho, wo))
    probe = torch.complex(rnd(P, n, n), rnd(P, n, n)).contiguous()
    kr = torch.polar(torch.ones(S - 1, n, device="cuda"), 0.5 * rnd(S - 1, n)).contiguous()
    kc = torch.polar(torch.ones(S - 1, n, device="cuda"), 0.5 * rnd(S - 1, n)).contiguous()
    pos = (torch.rand((B, 2), generator=g, device="cuda") * torch.tensor([ho - n - 2.0, wo - n - 2.0], device="cuda")
           + n // 2 + 1).contiguous()
    targets = (torch.rand((B, n, n), generator=g, device="cuda") * n).contiguous()
    return obj.contiguous(), probe, (kr, kc), pos, targets


def _run(obj, probe, prop, pos, targets):
    n = probe.shape[-1]
    idx = torch.arange(pos.shape[0], device="cuda")
    mask = torch.ones((n, n), device="cuda")
    loss, go, gp = ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, pos.shape[0], 100.0)
    out = ops.batch_forward(obj, probe, prop, pos, idx, targets, mask, pos.shape[0], 100.0)
    return float(loss), go.cpu().numpy(), gp.cpu().numpy(), out["intensity"].cpu().numpy()


@pytest.mark.parametrize("n,wo", [(64, 101), (96, 130), (128, 177)])
def test_wrapped_windows_match_interior_ones(n, wo):
    """Rolling the object and moving every position with it changes nothing but which columns
    wrap: the column paths agree to the rounding of a sum (the kernels' products are the same;
    only the order of the atomic additions differs, about 8 per pixel: 8 eps = 1e-6)."""
    ho = n + 23
    obj, probe, prop, pos, targets = _problem(n, 3, 2, 9, ho, wo)
    base = _run(obj, probe, prop, pos, targets)
    for shift in (-int(pos[:, 1].min()) + n // 2, wo // 2, int(wo - pos[:, 1].max().ceil() - n // 2)):
        p2 = pos.clone()
        p2[:, 1] = pos[:, 1] + shift  # integer shift: the fractional parts stay (up to its rounding, 2^-17 px)
        p2[:, 1] = torch.round(pos[:, 1]) + shift + (pos[:, 1] - torch.round(pos[:, 1]))
        got = _run(torch.roll(obj, shift, dims=2).contiguous(), probe, prop, p2.contiguous(), targets)
        # a position near 200 px holds its fraction to 2^-17: 1e-5 of phase at the band edge
        assert abs(got[0] - base[0]) < 1e-4 * abs(base[0])
        assert rel(got[3], base[3]) < 1e-4
        assert rel(np.roll(got[1], -shift, axis=2), base[1]) < 1e-4
        assert rel(got[2], base[2]) < 1e-4


@pytest.mark.parametrize("n,S", [(64, 2), (64, 30), (96, 9), (128, 13), (128, 14), (128, 15)])
def test_separable_propagators_match_the_full_array(n, S):
    """The separable factors (shared memory, or the L1 cache where they do not fit) against the
    product array: one extra rounding of each propagator value per slice (S 2^-23 relative)."""
    obj, probe, prop, pos, targets = _problem(n, S, 1, 5, n + 20, n + 31, seed=S)
    full = (prop[0][:, :, None] * prop[1][:, None, :]).contiguous()
    a, b = _run(obj, probe, prop, pos, targets), _run(obj, probe, full, pos, targets)
    tol = 4 * S * 2.0 ** -23
    assert abs(a[0] - b[0]) < tol * abs(b[0])
    for x, y in zip(a[1:], b[1:]):
        assert rel(x, y) < tol


@pytest.mark.parametrize("n,B", [(64, 1), (64, 149), (64, 700), (96, 310), (128, 150)])
def test_many_ctas_match_one_position_at_a_time(n, B):
    """A launch with several CTAs per SM and several positions per CTA against the sum of
    single-position launches (sums of B float32 terms in another order: sqrt(B) eps)."""
    obj, probe, prop, pos, targets = _problem(n, 2, 2, B, n + 40, n + 45, seed=B)
    loss, go, gp, inten = _run(obj, probe, prop, pos, targets)
    idx = torch.arange(B, device="cuda")
    mask = torch.ones((n, n), device="cuda")
    go2, gp2, l2 = torch.zeros_like(obj, dtype=torch.complex128), 0, 0.0
    for b in range(0, B, max(1, B // 7)):
        sel = idx[b:b + max(1, B // 7)]
        l, g, q = ops.batch_forward_adjoint(obj, probe, prop, pos, sel, targets, mask, B, 100.0)
        w = sel.numel() / B  # the loss scale carries 1 / batch
        l2, go2, gp2 = l2 + w * float(l), go2 + w * g.to(torch.complex128), gp2 + w * q.to(torch.complex128)
    assert abs(loss - l2) < 1e-6 * abs(l2)
    assert rel(go, go2.cpu().numpy()) < 4e-7 * max(4.0, B ** 0.5)
    assert rel(gp, gp2.cpu().numpy()) < 4e-7 * max(4.0, B ** 0.5)


@pytest.mark.parametrize("n,P", [(64, 1), (64, 3), (96, 2), (128, 1), (128, 2)])
def test_blocks_without_a_valid_first_position(n, P):
    """Three blocks of two positions: the second has only invalid indices (its probe-gradient
    partial must still be zero, whatever the workspace held), the third starts with one (its
    second position is then the one that writes the partial).  Against the valid positions alone,
    one by one: sums of three float32 terms, as above."""
    obj, probe, prop, pos, targets = _problem(n, 2, P, 6, n + 20, n + 23, seed=P)
    mask = torch.ones((n, n), device="cuda")
    torch.full((1 << 26,), float("nan"), device="cuda")  # what a fresh workspace may hold
    idx = torch.tensor([0, 1, 6, -1, 7, 5], device="cuda")
    loss, go, gp = ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, 6, 100.0, grid=3)
    assert ops.read_status(obj.device)["invalid_indices"] == 3
    l2, go2, gp2 = 0.0, 0, 0
    for b in (0, 1, 5):
        l, g, q = ops.batch_forward_adjoint(obj, probe, prop, pos, idx.new_tensor([b]), targets, mask, 6, 100.0)
        l2, go2, gp2 = l2 + float(l) / 6, go2 + g.to(torch.complex128) / 6, gp2 + q.to(torch.complex128) / 6
    assert abs(float(loss) - l2) < 1e-6 * abs(l2)
    assert rel(go.cpu().numpy(), go2.cpu().numpy()) < 1.6e-6
    assert rel(gp.cpu().numpy(), gp2.cpu().numpy()) < 1.6e-6
