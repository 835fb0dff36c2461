"""The marching convolution on planes of more than 2^31 input values (its piece
offsets stay within 32 bits as 16-byte pieces), against the one-plane form on
the same box, whose offsets are 64-bit: the last rows and columns, where an
offset in values would have wrapped."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_plane_of_more_than_2_31_values(gpu, monkeypatch):
    from voxelsim_fea_b200.learned import conv
    shape, cin, cout = (2, 5800, 5800), 64, 32
    assert shape[1] * shape[2] * cin > 2 ** 31
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.zeros(*shape, cin, device="cuda", dtype=torch.bfloat16)
    for rows in (slice(0, 64), slice(2890, 2930), slice(5700, 5800)):
        x[:, rows] = torch.randn(shape[0], rows.stop - rows.start, shape[2], cin, generator=g, device="cuda").bfloat16()
    w = (torch.randn(27, cout, cin, generator=g, device="cuda") / 40).bfloat16()
    monkeypatch.setenv("VOXFEA_CONV_FORM", "column")
    y = conv.conv3d_forward(x, w)
    monkeypatch.setenv("VOXFEA_CONV_FORM", "plane")
    ref = conv.conv3d_forward(x, w)
    assert torch.equal(y, ref)
    assert float(ref[:, 5750:].float().abs().max()) > 1
