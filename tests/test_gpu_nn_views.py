"""One convolution layer on views: inputs and output gradients that are not
contiguous, or contiguous but not on a 16-byte boundary of their storage, give
bit for bit the gradients of plain copies, with every gradient asked for and
with the bias' alone."""

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPE, CIN, COUT = (6, 10, 12), 16, 32


def _case():
    g = torch.Generator(device="cuda").manual_seed(1)
    new = lambda *d: torch.randn(*d, generator=g, device="cuda")  # noqa: E731
    return (new(*SHAPE, CIN).bfloat16(), new(27, COUT, CIN) / (27 * CIN) ** 0.5, new(COUT),
            new(*SHAPE, COUT).bfloat16())


def _grads(x, w, b, dy, which="xwb"):
    from voxelsim_fea_b200.learned import conv
    t = [v.detach().requires_grad_(k in which) for k, v in zip("xwb", (x, w, b))]
    y = conv.conv3d(*t)
    return [y.detach()] + list(torch.autograd.grad(y, [v for v in t if v.requires_grad], dy))


def _transposed(t):
    return t.transpose(0, 2).contiguous().transpose(0, 2)


def _shifted(t, k):
    flat = torch.zeros(t.numel() + k, dtype=t.dtype, device=t.device)
    flat[k:] = t.reshape(-1)
    return flat[k:].view(t.shape)


@pytest.mark.parametrize("which", ["xwb", "b"])
def test_non_contiguous(gpu, which):
    x, w, b, dy = _case()
    ref = _grads(x, w, b, dy, which)
    for got in (_grads(_transposed(x), w, b, dy, which), _grads(x, w, b, _transposed(dy), which)):
        for a, r in zip(got, ref):
            assert torch.equal(a, r)


@pytest.mark.parametrize("which", ["xwb", "b"])
def test_off_a_16_byte_boundary(gpu, which):
    x, w, b, dy = _case()
    ref = _grads(x, w, b, dy, which)
    for k in (1, 3, 4):
        assert _shifted(dy, k).is_contiguous() and _shifted(dy, k).data_ptr() % 16
        for got in (_grads(_shifted(x, k), w, b, dy, which), _grads(x, w, b, _shifted(dy, k), which),
                    _grads(x, _shifted(w.bfloat16(), k), b, dy, which)):
            for a, r in zip(got, ref):
                assert torch.equal(a, r.to(a.dtype))
