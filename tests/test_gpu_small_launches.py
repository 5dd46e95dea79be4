"""Launches whose shape follows the amount of work: results on both sides of each line, and that small (or
large) calls are not slower than the work they do."""
import numpy as np
import pytest
import torch

from quantem_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def device_us(f):
    """Device time of one call: 20 of them in a CUDA graph."""
    for _ in range(2):
        f()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        f()
    torch.cuda.current_stream().wait_stream(side)
    graph, best = torch.cuda.CUDAGraph(), float("inf")
    with torch.cuda.graph(graph):
        for _ in range(20):
            f()
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 50)
    return best


@pytest.mark.parametrize("shape", [(1, 100, 100), (3, 33, 47), (1, 447, 447), (1, 450, 445), (7, 190, 151), (2, 401, 520)])
@pytest.mark.parametrize("ntaps", [1, 3, 7, 33, 35])
@pytest.mark.parametrize("cplx", [True, False])
def test_blur_any_size(cuda_device, shape, ntaps, cplx):
    """Against FP64: two sums of ntaps float32 products, 2 (ntaps + 1) 2^-24 relative to the absolute sums."""
    rng = np.random.default_rng(sum(shape) + ntaps)
    x = rng.standard_normal(shape) + (1j * rng.standard_normal(shape) if cplx else 0)
    x = x.astype(np.complex64 if cplx else np.float32)
    taps = rng.uniform(0.1, 1.0, ntaps).astype(np.float32)
    taps = (taps + taps[::-1]) / taps.sum() / 2
    t = torch.tensor(x, device=cuda_device)
    got = ops._blur(t, torch.tensor(taps, device=cuda_device)).cpu().numpy()
    k = torch.tensor(taps.astype(np.float64))

    def blur(v):
        v = torch.tensor(v.astype(np.float64))[:, None]
        v = torch.nn.functional.conv2d(v, k.view(1, 1, -1, 1), padding=(ntaps // 2, 0))
        return torch.nn.functional.conv2d(v, k.view(1, 1, 1, -1), padding=(0, ntaps // 2))[:, 0].numpy()

    want, size = (blur(x.real) + 1j * blur(x.imag), blur(abs(x.real)) + blur(abs(x.imag))) if cplx else (blur(x), blur(abs(x)))
    assert np.all(np.abs(got - want) <= 2 * (ntaps + 1) * 2.0 ** -24 * size + 1e-30)


def test_small_blur_takes_less_than_a_large_one(cuda_device):
    """100 x 100 values against 510 x 516 (33 taps, complex): 16 tiles on 148 SMs took three quarters of the time
    of 272."""
    lib, times = _lib.lib(), []
    taps = torch.full((33,), 1 / 33, device="cuda")
    for H, W in ((100, 100), (510, 516)):
        x, o, tmp = (torch.randn(1, H, W, dtype=torch.complex64, device="cuda") for _ in range(3))
        times.append(device_us(lambda: lib.ptycho_obj_blur(ops._p(x), ops._p(o), ops._p(tmp), 1, H, W, 1, ops._p(taps), 33,
                                                           ops._stream())))
    assert times[0] < 0.6 * times[1], times


@pytest.mark.parametrize("nparts,count", [(1, 1), (7, 100), (444, 4096), (85, 65536), (86, 65536), (148, 65536),
                                          (148, 65537), (21, 16384), (22, 16384), (33, 1 << 18), (2, 3000001)])
def test_reduce_partials_any_shape(cuda_device, nparts, count):
    """Sums of nparts float32 values: nparts 2^-24 of the absolute sum."""
    g = torch.Generator(device="cuda").manual_seed(nparts)
    x = torch.randn(nparts, count, dtype=torch.complex64, device="cuda", generator=g)
    out = torch.full((count,), float("nan"), dtype=torch.complex64, device="cuda")
    _lib.check(_lib.lib().ptycho_reduce_partials(ops._p(x), ops._p(out), nparts, count, ops._stream()), "reduce")
    want, size = x.to(torch.complex128).sum(0), torch.view_as_real(x).abs().double().sum(0)
    err = torch.view_as_real(out.to(torch.complex128) - want).abs()
    assert bool((err <= nparts * 2.0 ** -24 * size).all())


def test_large_reductions_read_their_input_once(cuda_device):
    """Two partials of four million values: close to a copy of one (13 times a copy with the lanes)."""
    n = 1 << 22
    x, out = torch.randn(2, n, dtype=torch.complex64, device="cuda"), torch.empty(n, dtype=torch.complex64, device="cuda")
    copy = device_us(lambda: out.copy_(x[0]))
    t = device_us(lambda: _lib.lib().ptycho_reduce_partials(ops._p(x), ops._p(out), 2, n, ops._stream()))
    assert t < 4 * copy, (t, copy)


@pytest.mark.parametrize("n,per_sm", [(64, 3), (96, 2)])
def test_a_few_positions_more_than_blocks(cuda_device, n, per_sm):
    """Six positions more than resident blocks cost about one position on an SM of its own, half of a full round
    or less (0.9 of one when the six longer blocks shared two SMs)."""
    from tests.test_gpu_batch_paths import _problem

    times = []
    for B in (ops.resident_ctas(n), ops.resident_ctas(n) + 6):
        assert ops.resident_ctas(n) == per_sm * ops.sm_count()
        obj, probe, prop, pos, targets = _problem(n, 16, 1, B, n + 150, n + 150)
        idx, mask = torch.arange(B, device="cuda"), torch.ones((n, n), device="cuda")
        ph, go, gp = ops.fft2(probe), torch.zeros_like(obj), torch.empty_like(probe)
        times.append(device_us(lambda: ops.batch_forward_adjoint(obj, probe, prop, pos, idx, targets, mask, B, 100.0,
                                                                 probe_hat=ph, grad_obj=go, grad_probe=gp)))
    assert times[1] < 1.75 * times[0], times
