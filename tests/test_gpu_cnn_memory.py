"""What a training step of the network holds on the device while its backward runs."""
import weakref

import pytest
import torch

from quantem_b200.core.ml import cnn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skip", [True, False])
def test_backward_gives_forward_buffers_back(cuda_device, monkeypatch, skip):
    """At the last layer of the backward only the top encoder level's forward buffers are left: with two
    levels about a quarter of all (a decoder level holds about as much as its encoder level and the skip,
    each deeper level half of the one above).  The same on the first pass of a shape and on later ones."""
    net = cnn.CNN2d(8, 4, start_filters=32, num_layers=2, use_skip_connections=skip)
    net.train()
    x = torch.randn(2, 8, 128, 128, device=cuda_device)
    bases, alive = {}, []
    init, call = cnn._Buf.__init__, cnn._Run.call

    def seen_init(self, base, *args):
        init(self, base, *args)
        bases[id(base)] = weakref.ref(base)

    def seen_call(self, name, *args):
        if name == "ptycho_cnn_conv_backward":
            alive.append(sum(t.numel() for t in (r() for r in bases.values()) if t is not None))
        return call(self, name, *args)

    monkeypatch.setattr(cnn._Buf, "__init__", seen_init)
    monkeypatch.setattr(cnn._Run, "call", seen_call)
    for _ in range(3):
        bases.clear()
        alive.clear()
        net(x).square().mean().backward()
        assert alive[-1] < 0.4 * alive[0], alive
        assert all(a >= b for a, b in zip(alive, alive[1:])), alive


def test_training_step_peak(cuda_device):
    """Peak of a training step over the network's own tensors, from its parts: every forward buffer once, the
    largest layer's scratch (BF16 gradients, patches or their FP32 gradients in one place) and, at the two
    widest layers, the FP32 gradients that pass between them."""
    net = cnn.CNN2d(8, 8, start_filters=32, num_layers=2)
    net.train()
    B, H = 2, 256
    R = B * H * H
    x = torch.randn(B, 8, H, H, device=cuda_device)
    for _ in range(2):
        net.flat.grad = None
        net(x).square().mean().backward()
    net.flat.grad = None
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    base = torch.cuda.memory_allocated()
    y = net(x)
    held = torch.cuda.memory_allocated() - base
    torch.cuda.reset_peak_memory_stats()
    y.square().mean().backward()
    peak = torch.cuda.max_memory_allocated() - base
    # the widest layer: the decoder's first 3x3 convolution, 64 -> 32 channels at full size
    scratch = R * (32 * 2 + 9 * 64 * 4)
    between = R * 4 * (64 + 32 + 32) + R * 4 * 8 * 6
    assert peak < held + scratch + between, (peak / R, held / R, scratch / R)
