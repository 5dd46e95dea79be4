"""The launch autotuner keeps a partition for the question it was asked."""
import pytest
import torch

from tests.test_gpu_multi import SPECS, _problems

pytestmark = pytest.mark.gpu


def test_partitions_are_kept_per_total_and_kind_of_propagators(cuda_device):
    """A tuning over a few CTAs must not fix the partition of a later one over the device, nor one with
    separable propagators that of the whole arrays (they take other shared memory and code)."""
    from quantem_b200 import multi

    probs, cache = _problems(cuda_device, SPECS), {}
    few = multi.autotune_grids(probs, total=6, cache=cache)
    all_ = multi.autotune_grids(probs, cache=cache)
    assert sum(few) <= 12 + 4 and len(cache) == 2  # at most twice the total, and one CTA each at least
    assert multi.autotune_grids(probs, total=6, cache=cache) == few
    assert multi.autotune_grids(probs, cache=cache) == all_ and len(cache) == 2
    for p in probs:
        S, n = p.obj.shape[0], p.probe.shape[-1]
        if isinstance(p.prop, (tuple, list)):
            p.prop = (p.prop[0][:, :, None] * p.prop[1][:, None, :]).contiguous()
        else:
            p.prop = (torch.ones(S - 1, n, dtype=torch.complex64, device=cuda_device),) * 2
    multi.autotune_grids(probs, total=6, cache=cache)
    assert len(cache) == 3
