"""Small windows run several CTAs per SM; where the scratch of so many does not fit on the device the
launch takes one per SM, which is what earlier memory plans were made for."""
import pytest
import torch

from quantem_b200 import ops
from tests.conftest import rel
from tests.test_gpu_batch_paths import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 96])
def test_less_memory_than_the_resident_ctas_take(cuda_device, monkeypatch, n):
    B = 2 * ops.resident_ctas(n)
    sms = ops.sm_count()
    obj, probe, prop, pos, targets = _problem(n, 2, 2, B, n + 20, n + 25)
    idx, mask = torch.arange(B, device="cuda"), torch.ones((n, n), device="cuda")

    def run():
        return ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, B, 100.0)

    want = run()
    limit = sms * (2 * 2 + 2 + 1) * n * n  # the scratch of one CTA per SM
    ensure, grids, refused = ops.Workspace.ensure, [], []
    monkeypatch.setattr(ops.workspace(obj.device), "refused", None)

    def small(self, scratch_elems, partial_elems, grid):
        if scratch_elems > limit:
            refused.append(grid)
            raise torch.OutOfMemoryError("no memory")
        grids.append(grid)
        return ensure(self, scratch_elems, partial_elems, grid)

    monkeypatch.setattr(ops.Workspace, "ensure", small)
    for k in (1, 2):  # the second launch does not try the larger scratch again
        got = run()
        assert grids == [sms] * k and refused == [B // 2]
        assert abs(float(got[0]) - float(want[0])) < 1e-6 * abs(float(want[0]))
        for a, b in zip(got[1:], want[1:]):  # sums of the same terms in another order
            assert rel(a.cpu().numpy(), b.cpu().numpy()) < 4e-7 * B ** 0.5


def test_partition_of_several_datasets(cuda_device, monkeypatch):
    """A multi-dataset launch whose scratch does not fit takes one CTA per SM, and does not try again."""
    from quantem_b200 import multi
    from tests.test_gpu_multi import _problems

    probs = _problems(cuda_device, [(20, 3, 2), (22, 2, 2)])
    grids = multi.default_grids(probs)
    assert sum(grids) == ops.resident_ctas(64)
    objs, probes = [p.obj.detach().contiguous() for p in probs], [p.probe.detach().contiguous() for p in probs]
    want = multi.multi_forward_adjoint(probs, objs, probes, grids)
    small = multi.default_grids(probs, ops.sm_count())
    limits = {}
    for p, g in zip(probs, small):
        n, S, P, *_ = p.signature()
        limits[id(p.ws)] = g * (P * S + P + 1) * n * n
    for p in probs:
        p.ws.scratch = p.ws.partials = None
    ensure, refused = ops.Workspace.ensure, []

    def limited(self, scratch_elems, partial_elems, grid):
        if scratch_elems > limits[id(self)]:
            refused.append(grid)
            raise torch.OutOfMemoryError("no memory")
        return ensure(self, scratch_elems, partial_elems, grid)

    monkeypatch.setattr(ops.Workspace, "ensure", limited)
    for _ in range(2):
        got = multi.multi_forward_adjoint(probs, objs, probes, grids)
        assert len(refused) == 1
        assert [p.ws.scratch.numel() for p in probs] == [limits[id(p.ws)] for p in probs]
        for p, g, w in zip(probs, got, want):
            assert abs(float(g[0]) - float(w[0])) < 1e-6 * abs(float(w[0]))
            for a, b in zip(g[1:], w[1:]):  # sums of the same terms in another order
                assert rel(a.cpu().numpy(), b.cpu().numpy()) < 4e-7 * p.num_gpts ** 0.5
    for p in probs:  # nothing smaller to fall back to
        limits[id(p.ws)] = 0
    with pytest.raises(torch.OutOfMemoryError):
        multi.multi_forward_adjoint(probs, objs, probes, small)


def test_default_partition_asks_no_driver(cuda_device, monkeypatch):
    """The driver's free-memory query waits for the other processes of the host, up to 130 ms."""
    from quantem_b200 import multi
    from tests.test_gpu_multi import _problems

    probs = _problems(cuda_device, [(20, 3, 2)])

    def query(*a, **k):
        raise AssertionError("cudaMemGetInfo")

    monkeypatch.setattr(torch.cuda, "mem_get_info", query)
    multi.default_grids(probs)
