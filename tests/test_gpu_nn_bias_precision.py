"""Precision of the convolution's bias gradient against FP64 on normal values.
A thread adds c = ceil(voxels / (148 blocks x voxels of a block)) values in FP32;
with sums of the threads and of the blocks in FP64 and one rounding of each
block's sum, the rounding errors add up to about 2^-25 (0.3 c + 0.6) of the
result (c <= 14 here: below 1.5e-7 / 2); 1e-7 is allowed.  Not less exact than a
pairwise FP32 sum."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cout", [16, 32, 64])
@pytest.mark.parametrize("shape", [(20, 28, 36), (36, 52, 68)])
def test_bias_gradient_against_fp64(gpu, cout, shape):
    from voxelsim_fea_b200.learned import conv
    worst = 0.0
    for seed in range(4):
        g = torch.Generator(device="cuda").manual_seed(100 * seed + cout)
        dy = torch.randn(*shape, cout, generator=g, device="cuda").bfloat16()
        ref = dy.double().sum(dim=(0, 1, 2))
        worst = max(worst, float((conv.conv3d_backward_bias(dy).double() - ref).norm() / ref.norm()))
    assert worst <= 1e-7
