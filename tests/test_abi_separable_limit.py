"""How many slices the separable propagators are accepted for (no GPU needed)."""
import ctypes

import pytest


@pytest.mark.parametrize("n,most", [(64, 176), (96, 73), (128, 15)])
def test_slices_with_separable_propagators(n, most):
    from quantem_b200 import _lib

    lib = _lib.lib()
    a = _lib.BatchArgs()
    d = ctypes.c_void_p(256)  # never dereferenced: every call below fails validation
    for f in ("obj", "probe_hat", "prop_r", "prop_c", "positions", "batch_idx", "targets", "mask", "loss_part"):
        setattr(a, f, d)
    a.n, a.P, a.B, a.Ho, a.Wo, a.npos, a.grid = n, 1, 4, 256, 256, 4, 4
    a.loss_type = 9  # refused after the slices are accepted
    a.S = most
    assert lib.ptycho_forward_loss(ctypes.byref(a), None) == 1 and "loss type" in _lib.last_error()
    a.S = most + 1
    assert lib.ptycho_forward_loss(ctypes.byref(a), None) == 2
    assert f"up to {most} slices" in _lib.last_error()

