"""Batch norms of many rows (separate launches over all SMs) and of fewer (one cluster launch): both sides
of the line between them, against FP64."""
import pytest
import torch

from quantem_b200.core.ml import kernels as kk

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _data(R, C, ld, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(R, ld, device="cuda", generator=g)[:, :C] * 0.7 + 0.4
    dy = torch.randn(R, ld, device="cuda", generator=g)[:, :C]
    ga, be = (torch.rand(C, device="cuda", generator=g) + 0.5 for _ in range(2))
    rm, rv = torch.randn(C, device="cuda", generator=g), torch.rand(C, device="cuda", generator=g) + 0.5
    return x, dy, ga, be, rm, rv


@pytest.mark.parametrize("R", [16383, 16384, 32767, 32768, 33001, 70003])
@pytest.mark.parametrize("C,ld", [(1, 8), (7, 8), (32, 32), (100, 104), (256, 256), (300, 304)])
@pytest.mark.parametrize("training", [True, False])
def test_batch_norm_rows(cuda_device, R, C, ld, training):
    x, dy, ga, be, rm, rv = _data(R, C, ld, R + C)
    rm0, rv0 = rm.double(), rv.double()
    mean, rstd = torch.empty(C, device="cuda"), torch.empty(C, device="cuda")
    work = torch.full((2 * 592 * C,), float("nan"), device="cuda", dtype=torch.float64)
    y = torch.empty(R, ld, device="cuda", dtype=torch.bfloat16)[:, :C]
    kk.bn_forward(x, ga, be, rm, rv, 0.1, 1e-5, training, mean, rstd, work, y)
    xd = x.double()
    mu, var = (xd.mean(0), xd.var(0, unbiased=False)) if training else (rm0, rv0)
    rs = 1.0 / torch.sqrt(var + 1e-5)
    # float runs of at most 64 terms, then doubles: 64 eps of the mean size, a few roundings behind it
    assert float((mean.double() - mu).abs().max()) < 64 * EPS * 2
    assert float(((rstd.double() - rs) / rs).abs().max()) < 128 * EPS * 2
    if training:
        assert float((rm.double() - (0.9 * rm0 + 0.1 * mu)).abs().max()) < 64 * EPS * 4
        assert float((rv.double() - (0.9 * rv0 + 0.1 * xd.var(0))).abs().max()) < 64 * EPS * 4
    want = (xd - mu) * rs * ga.double() + be.double()
    assert float(((y.double() - want).abs() / (want.abs() + 0.1)).max()) < 2.0 ** -8  # BF16, an ulp flip
    dg, db = torch.empty(C, device="cuda"), torch.empty(C, device="cuda")
    dz = torch.empty(R, ld, device="cuda")[:, :C]
    work.fill_(float("nan"))
    kk.bn_backward(dy, x, ga, mean, rstd, training, 1, dg, db, work, dz32=dz)
    xh, dyd = (xd - mean.double()) * rstd.double(), dy.double()
    scale = dyd.abs().sum(0) * EPS * 64  # runs of 64 float terms
    assert bool(((db.double() - dyd.sum(0)).abs() <= scale).all())
    assert bool(((dg.double() - (dyd * xh).sum(0)).abs() <= 4 * (dyd * xh).abs().sum(0) * EPS * 64).all())
    g = (dyd - dyd.mean(0) - xh * (dyd * xh).mean(0)) if training else dyd
    g = g * ga.double() * rstd.double() * (x > 0)
    assert float((dz.double() - g).abs().max()) < 64 * EPS * float(g.abs().max())


@pytest.mark.parametrize("R,C", [(16384, 32), (40000, 24)])
def test_activation_backward_rows(cuda_device, R, C):
    x, dy, *_ = _data(R, C, C, 3)
    work = torch.empty(2 * 592 * C, device="cuda", dtype=torch.float64)
    dz = torch.empty(R, C, device="cuda")
    kk.bn_backward(dy, x, None, None, None, True, 1, None, None, work, dz32=dz)
    assert torch.equal(dz, torch.where(x > 0, dy, torch.zeros_like(dy)))


def test_small_workspace_takes_the_cluster_launch(cuda_device):
    """The statistics are those of the wide launches: the same float runs, their doubles added in another order."""
    R, C = 50000, 40
    x, _, ga, be, rm, rv = _data(R, C, C, 9)
    out = []
    for elems in (2 * C, 2 * 592 * C):
        mean, rstd = torch.empty(C, device="cuda"), torch.empty(C, device="cuda")
        y = torch.empty(R, C, device="cuda", dtype=torch.bfloat16)
        kk.bn_forward(x, ga, be, rm.clone(), rv.clone(), 0.1, 1e-5, True, mean, rstd,
                      torch.empty(elems, device="cuda", dtype=torch.float64), y)
        out.append((mean, rstd))
    for a, b in zip(*out):
        assert float(((a - b) / b).abs().max()) <= 2 * EPS


def test_many_rows_use_the_device(cuda_device):
    """262144 x 32 values: the passes stay within a few copies of the same data (one cluster per eight channels,
    32 blocks on 148 SMs, took 20 times the copy backward and 7 times forward)."""
    R, C = 262144, 32
    x, dy, ga, be, rm, rv = _data(R, C, C, 1)
    mean, rstd, dg, db = (torch.empty(C, device="cuda") for _ in range(4))
    y, y2 = torch.empty(R, C, device="cuda", dtype=torch.bfloat16), torch.empty_like(x)
    work = torch.empty(2 * 592 * C, device="cuda", dtype=torch.float64)

    def us(f):
        best = float("inf")
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                f()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 100)
        return best

    copy = us(lambda: y2.copy_(x))
    fwd = us(lambda: kk.bn_forward(x, ga, be, rm, rv, 0.1, 1e-5, True, mean, rstd, work, y))
    bwd = us(lambda: kk.bn_backward(dy, x, ga, mean, rstd, True, 1, dg, db, work, dz16=y))
    assert fwd < 5 * copy and bwd < 9 * copy, (copy, fwd, bwd)


@pytest.mark.parametrize("R", [64, 40000])
def test_running_variance_without_mean_is_ignored(cuda_device, R):
    """Batch statistics with a running variance but no running mean: nothing is updated, as without both."""
    x, _, ga, be, _, rv = _data(R, 24, 24, R)
    work = torch.empty(2 * 592 * 24, device="cuda", dtype=torch.float64)
    outs = []
    for var in (None, rv.clone()):
        mean, rstd = torch.empty(24, device="cuda"), torch.empty(24, device="cuda")
        y = torch.empty(R, 24, device="cuda", dtype=torch.bfloat16)
        kk.bn_forward(x, ga, be, None, var, 0.1, 1e-5, True, mean, rstd, work, y)
        outs.append((mean, rstd, y))
    assert all(torch.equal(a, b) for a, b in zip(*outs)) and torch.equal(var, rv)
