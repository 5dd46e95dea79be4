"""Host threads that call the same kernels with different shared-memory needs at the same time:
no thread's launch depends on what another asks for (a kernel's shared-memory bound belongs to the
device, and ctypes lets the calls run side by side)."""
import ctypes
import threading

import pytest
import torch

from quantem_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _side_by_side(calls, reps=3000):
    """Every call in a thread and on a stream of its own, reps times; the error codes that are not 0."""
    bad, start = [], threading.Barrier(len(calls))

    def work(call):
        st = torch.cuda.Stream()
        start.wait()
        for _ in range(reps):
            rc = call(ctypes.c_void_p(st.cuda_stream))
            if rc:
                bad.append((rc, _lib.last_error()))
                break
        st.synchronize()

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return bad


def _c64(*shape):
    return torch.randn(*shape, dtype=torch.complex64, device="cuda")


def test_orthogonalize_side_by_side(cuda_device):
    lib = _lib.lib()

    def call(P, n):
        we = lib.ptycho_probe_ortho_work_elems(P, n * n)
        x, o, g, w = _c64(P, n, n), _c64(P, n, n), _c64(P, n, n), _c64(we)

        def f(st):
            rc = lib.ptycho_probe_orthogonalize(ops._p(x), ops._p(o), P, n * n, ops._p(w), we, st)
            return rc or lib.ptycho_probe_orthogonalize_vjp(ops._p(x), ops._p(o), ops._p(g), P, n * n, ops._p(w), we, st)
        return f

    torch.cuda.synchronize()
    assert _side_by_side([call(1, 64), call(4, 128), call(2, 96)]) == []


def test_object_filters_side_by_side(cuda_device):
    lib = _lib.lib()

    def call(H, W, ntaps):
        x, o, tmp, mu = _c64(1, H, W), _c64(1, H, W), _c64(2, H, W), _c64(2)
        env = torch.ones(H, W, device="cuda")
        taps = torch.full((ntaps,), 1.0 / ntaps, device="cuda")

        def f(st):
            rc = lib.ptycho_obj_butterworth(ops._p(x), ops._p(o), 1, H, W, 0, ops._p(env), ops._p(tmp), ops._p(mu), st)
            return rc or lib.ptycho_obj_blur(ops._p(x), ops._p(o), ops._p(tmp), 1, H, W, 1, ops._p(taps), ntaps, st)
        return f

    torch.cuda.synchronize()
    assert _side_by_side([call(40, 2100, 3), call(64, 64, 33), call(30, 600, 21)]) == []


@pytest.mark.parametrize("n", [64, 96, 128])
def test_forward_side_by_side(cuda_device, n):
    """The forward kernel with and without the intensities (the sum's tile in the output or in shared
    memory) and with few and many slices (separable factors in shared memory)."""
    lib = _lib.lib()
    keep = []

    def call(S, want):
        B, side = 4, n + 12
        obj, probe = _c64(S, side, side), _c64(2, n, n)
        prop = (_c64(S - 1, n), _c64(S - 1, n))
        pos = torch.full((B, 2), side / 2.0, device="cuda")
        idx, mask = torch.arange(B, device="cuda"), torch.ones(n, n, device="cuda")
        targets = torch.ones(B, n, n, device="cuda")
        out = torch.empty(B, n, n, device="cuda") if want else None
        geom = ops._check_batch_inputs(obj, probe, prop, pos, idx, targets, mask)
        a = ops._batch_args(geom, obj, probe, prop, pos, idx, targets, mask, B, "l2_amplitude", 1.0, 1.0,
                            out_intensity=out, variant="serial")
        part, status = torch.zeros(B, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        a.grid, a.loss_part, a.status = B, part.data_ptr(), status.data_ptr()
        keep.append((obj, probe, prop, pos, idx, mask, targets, out, part, status))
        return lambda st: lib.ptycho_forward_loss(ctypes.byref(a), st)

    torch.cuda.synchronize()
    assert _side_by_side([call(2, True), call(6, False), call(4, True)]) == []
