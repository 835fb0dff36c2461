"""Precision of the convolution's weight gradient against FP64.  The MMA's FP32
accumulators truncate, so a partial sum of L rows of 16 voxels loses about
(2/3) L ulp of itself; with 148 partials of one warp each (256 voxels = 16 rows a
tile) L is 16 ceil(tiles / 148), and 2^-24 L of the gradient's norm is allowed
for every pair of channels."""

import pytest
import torch

pytestmark = pytest.mark.gpu

PAIRS = [(16, 16), (16, 32), (32, 16), (32, 32), (32, 64), (64, 32), (64, 64)]


@pytest.mark.parametrize("cin,cout", PAIRS)
@pytest.mark.parametrize("shape", [(36, 52, 68), (50, 61, 83)])
def test_weight_gradient_against_fp64(gpu, cin, cout, shape):
    from voxelsim_fea_b200.learned import conv
    Z, Y, X = shape
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.relu(torch.randn(*shape, cin, generator=g, device="cuda")).bfloat16()
    dy = torch.randn(*shape, cout, generator=g, device="cuda").bfloat16()
    dw = conv.conv3d_backward_weight(x, dy)
    tiles = -(-X // 16) * -(-Y // 8) * -(-Z // 2)
    tol = 16 * -(-tiles // 148) * 2.0 ** -24
    xp = torch.nn.functional.pad(x.permute(3, 0, 1, 2), (1, 1, 1, 1, 1, 1))
    dyd = dy.double().reshape(-1, cout)
    err = ref = 0.0
    for t in (0, 4, 13, 17, 26):
        a = xp[:, t // 9:t // 9 + Z, t // 3 % 3:t // 3 % 3 + Y, t % 3:t % 3 + X].reshape(cin, -1).double()
        r = (a @ dyd).T
        err += float(((dw[t].double() - r) ** 2).sum())
        ref += float((r ** 2).sum())
    assert (err / ref) ** 0.5 <= tol
