"""The marching convolution on boxes where its columns hold several planes (full
ones and a shorter last one, partial tiles in x and y) against the one-plane
form, which the other tests compare with the oracle; both sum the same products
in FP32, so 1e-6 of the result's norm.  And the bias
gradient against FP64. """

import pytest
import torch

pytestmark = pytest.mark.gpu

PAIRS = [(16, 16), (16, 32), (32, 16), (32, 32), (32, 64), (64, 32), (64, 64)]


@pytest.mark.parametrize("cin,cout", PAIRS)
@pytest.mark.parametrize("shape", [(37, 50, 100), (64, 84, 61), (3, 200, 200)])
def test_columns_of_planes(gpu, monkeypatch, cin, cout, shape):
    from voxelsim_fea_b200.learned import conv
    torch.manual_seed(cin + 3 * cout)
    x = torch.randn(*shape, cin, device="cuda").to(torch.bfloat16)
    w = (torch.randn(27, cout, cin, device="cuda") / (27 * cin) ** 0.5).to(torch.bfloat16)
    b = torch.randn(cout, device="cuda")
    skip = torch.randn(*shape, cout, device="cuda").to(torch.bfloat16)
    monkeypatch.setenv("VOXFEA_CONV_FORM", "plane")
    ref = conv.conv3d_forward(x, w, bias=b, skip=skip, relu=True, out_f32=True)
    for form in ("column", ""):
        monkeypatch.setenv("VOXFEA_CONV_FORM", form)
        y = conv.conv3d_forward(x, w, bias=b, skip=skip, relu=True, out_f32=True)
        assert float((y - ref).norm() / ref.norm()) < 1e-6
        assert float((y - ref).abs().max()) < 1e-4


@pytest.mark.parametrize("n,cout", [(1, 16), (7, 64), (255, 32), (36 * 52 * 68, 32), (100001, 64)])
def test_bias_gradient(gpu, n, cout):
    from voxelsim_fea_b200.learned import conv
    torch.manual_seed(n)
    dy = torch.randn(1, 1, n, cout, device="cuda").to(torch.bfloat16)
    db = conv.conv3d_backward_bias(dy)
    ref = dy.double().sum(dim=(0, 1, 2))
    assert db.dtype == torch.float32 and db.shape == (cout,)
    # FP32 sums of n values of size 1: a few ulp of sqrt(n) .. n
    assert float((db.double() - ref).abs().max()) <= 1e-6 * float(dy.double().abs().sum(dim=(0, 1, 2)).max())
