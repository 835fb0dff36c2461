"""The bias gradient of a convolution layer is itself differentiable in the
output gradient (it is their sum), as a second derivative needs."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_bias_gradient_is_differentiable(gpu):
    from voxelsim_fea_b200.learned import conv
    g = torch.Generator(device="cuda").manual_seed(1)
    new = lambda *d: torch.randn(*d, generator=g, device="cuda")  # noqa: E731
    x, w = new(6, 10, 12, 16).bfloat16(), new(27, 32, 16) / 20
    b, dy = new(32).requires_grad_(), new(6, 10, 12, 32).bfloat16().requires_grad_()
    y = conv.conv3d(x, w, b)
    (db,) = torch.autograd.grad(y, b, dy, create_graph=True)
    v = torch.arange(32, device="cuda", dtype=torch.float32)
    (g2,) = torch.autograd.grad((db * v).sum(), dy)
    assert torch.equal(g2, v.to(torch.bfloat16).expand(dy.shape))
