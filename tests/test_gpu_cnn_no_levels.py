"""A network without encoder levels (num_layers = 0: bottleneck and output convolution) trains."""
import pytest
import torch
import torch.nn.functional as F

from quantem_b200.core.ml.cnn import CNN2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_batchnorm", [False, True])
def test_gradients_without_levels(cuda_device, use_batchnorm):
    """Against FP64 autograd.  About eight BF16 roundings (2^-9 each) lie between the weights and their
    gradients: 2^-9 x 8, doubled for the batch norms; the smooth activation has no masks that flip."""
    net = CNN2d(8, 3, start_filters=16, num_layers=0, use_batchnorm=use_batchnorm, activation="softplus",
                final_activation="identity", seed=3)
    net.train()
    g = torch.Generator().manual_seed(1)
    x, dy = torch.randn(2, 8, 24, 20, generator=g), torch.randn(2, 3, 24, 20, generator=g)
    sd = {k: v.detach().cpu().double().requires_grad_(v.is_floating_point() and "running" not in k)
          for k, v in net.state_dict().items()}
    net(x.to(cuda_device)).backward(dy.to(cuda_device))
    got = net.named_gradients()

    def conv(h, name):
        return F.conv2d(F.pad(h, (1, 1, 1, 1), mode="circular"), sd[name + ".weight"], sd[name + ".bias"])

    h, step = x.double(), 3 if use_batchnorm else 2
    for j in range(2):
        h = F.softplus(conv(h, f"bottleneck.block.{step * j}"))
        if use_batchnorm:
            p = f"bottleneck.block.{step * j + 2}"
            h = F.batch_norm(h, None, None, sd[p + ".weight"], sd[p + ".bias"], training=True)
    conv(h, "final_conv.block.0").backward(dy.double())
    checked = 0
    for k, v in got.items():
        want = sd[k].grad
        if want is None or (use_batchnorm and k.endswith("bias") and float(want.abs().max()) < 1e-9):
            continue  # a bias before a batch norm has no gradient
        err = float((v.cpu().double() - want).norm() / want.norm())
        assert err < (2 if use_batchnorm else 1) * 2.0 ** -6, (k, err)
        checked += 1
    assert checked >= 6
