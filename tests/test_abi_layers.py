"""The whole-layer entry points of the network refuse bad arguments before their first launch (no
GPU needed: every call below fails validation, nothing is dereferenced)."""
import ctypes

import pytest

INVALID = 1
P = ctypes.c_void_p(4096)     # aligned, never dereferenced
ODD = ctypes.c_void_p(4104)   # 8-byte aligned only
F = ctypes.c_float

# argument names in the order of include/ptycho_b200.h, with values that pass every check
CALLS = {
    "ptycho_cnn_conv_forward": dict(
        x=P, ldx=16, B=2, H=4, W=4, C=16, w=P, co=8, bias=P, act=1, gamma=P, beta=P, run_mean=P, run_var=P,
        momentum=F(0.1), eps=F(1e-5), training=1, mean=P, rstd=P, col=P, r=P, out=P, ldo=8, stream=None),
    "ptycho_cnn_conv_backward": dict(
        dy=P, lddy=8, x=P, ldx=16, B=2, H=4, W=4, C=16, w=P, r=P, co=8, gamma=P, mean=P, rstd=P, training=1, act=1,
        dw=P, db=P, dgamma=P, dbeta=P, dz=P, ldz=8, col=P, dcol=P, dx=P, lddx=16, dx_accumulate=0, stream=None),
    "ptycho_cnn_up_forward": dict(
        y=P, ldy=16, B=2, H=4, W=4, ci=16, co=8, wt=P, bt=P, w1=P, b1=P, gamma=P, beta=P, run_mean=P, run_var=P,
        momentum=F(0.1), eps=F(1e-5), training=1, mean=P, rstd=P, colT=P, t=P, r=P, out=P, ldo=8, stream=None),
    "ptycho_cnn_up_backward": dict(
        dup=P, lddup=8, y=P, ldy=16, t=P, r=P, B=2, H=4, W=4, ci=16, co=8, wt=P, w1=P, gamma=P, mean=P, rstd=P,
        training=1, dwt=P, dbt=P, dw1=P, db1=P, dgamma=P, dbeta=P, dz=P, ldz=8, dt=P, dcolT=P, work=P,
        work_elems=32, dy=P, stream=None),
}
SIZES = [dict(B=0), dict(H=0), dict(W=-1), dict(co=0), dict(B=1 << 15, H=1 << 15, W=4),
         dict(B=1 << 30, H=1 << 30, W=1 << 30)]
# running statistics: wanted without the batch's, the variance also with the mean
NO_STATISTICS = [dict(training=0, run_mean=None), dict(training=0, run_var=None), dict(training=1, run_var=None),
                 dict(training=0, run_mean=None, run_var=None)]
BAD = {
    "ptycho_cnn_conv_forward": SIZES + [dict(C=0), dict(C=12), dict(ldx=8), dict(ldo=7), dict(act=-1), dict(act=7)] + [
        {k: None} for k in ("x", "w", "col", "r", "beta", "mean", "rstd")] + [
        {k: ODD} for k in ("x", "w", "col")] + NO_STATISTICS,
    "ptycho_cnn_conv_backward": SIZES + [dict(C=0), dict(C=12), dict(lddy=7), dict(ldx=8), dict(ldz=7), dict(ldz=12),
                                         dict(lddx=15), dict(lddx=8), dict(act=-1), dict(act=7)] + [
        {k: None} for k in ("dy", "x", "w", "r", "mean", "rstd", "dw", "dgamma", "dbeta", "dz", "col", "dcol")] + [
        {k: ODD} for k in ("x", "w", "dz", "col", "dcol", "dx")],
    "ptycho_cnn_up_forward": SIZES + [dict(ci=0), dict(ci=12), dict(ldy=8), dict(ldo=7),
                                      dict(B=1 << 14, H=1 << 15, W=1)] + [
        {k: None} for k in ("y", "wt", "w1", "beta", "mean", "rstd", "colT", "t", "r", "out")] + [
        {k: ODD} for k in ("y", "wt", "w1", "t")] + NO_STATISTICS,
    "ptycho_cnn_up_backward": SIZES + [dict(ci=0), dict(ci=12), dict(lddup=7), dict(ldy=8), dict(ldz=7), dict(ldz=12),
                                       dict(work_elems=31), dict(B=1 << 14, H=1 << 15, W=1)] + [
        {k: None} for k in ("dup", "y", "t", "r", "wt", "w1", "mean", "rstd", "dwt", "dbt", "dw1", "dgamma", "dbeta", "dz",
                            "dt", "dcolT", "work", "dy")] + [
        {k: ODD} for k in ("y", "t", "wt", "w1", "dz", "dcolT")],
}


@pytest.mark.parametrize("name", CALLS)
def test_layer_calls_refuse_bad_arguments(name):
    from quantem_b200 import _lib

    fn = getattr(_lib.lib(), name)
    assert len(fn.argtypes) == len(CALLS[name])
    for bad in BAD[name]:
        assert fn(*{**CALLS[name], **bad}.values()) == INVALID, bad
        assert name.removeprefix("ptycho_cnn_").split("_")[0] in _lib.last_error() or "bn_" in _lib.last_error() or (
            "workspace" in _lib.last_error()), (bad, _lib.last_error())


def test_batch_norm_backward_still_refuses_missing_buffers():
    """The checks that the batch-norm entry points shared with the layer calls."""
    from quantem_b200 import _lib

    lib = _lib.lib()
    for mean, rstd, dg, db in ((None, P, P, P), (P, None, P, P), (P, P, None, P), (P, P, P, None)):
        assert lib.ptycho_cnn_bn_backward(P, 8, P, 8, 16, 8, P, mean, rstd, 1, 0, dg, db, P, 64, P, None, 8, None) == INVALID
    assert lib.ptycho_cnn_bn_backward(P, 8, P, 8, 16, 8, P, P, P, 1, 0, P, P, P, 15, P, None, 8, None) == INVALID
    assert lib.ptycho_cnn_bn_forward(P, 8, 16, 8, P, None, P, P, F(0.1), F(1e-5), 1, P, P, P, 64, P, 8, None) == INVALID
    assert lib.ptycho_cnn_bn_forward(P, 8, 16, 8, P, P, None, P, F(0.1), F(1e-5), 0, P, P, P, 64, P, 8, None) == INVALID
