"""vf_apply_noalloc on very long grids one voxel thick, with more tiles than blocks
may be launched (32,768): the gather form takes them -- against a plain FP64
evaluation, 1e-13 of the largest value."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1_030_000, 1, 1), (1_030_000, 1, 2)])
def test_more_tiles_than_blocks(gpu, dims):
    import torch
    from oracle import hex8
    from voxelsim_fea_b200 import _lib
    nx, ny, nz = dims
    assert (nx + 31) // 31 > 32768                       # tiles of 31 x 7 nodes, whole columns
    rng = np.random.default_rng(nz)
    nn, ne = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    E = rng.uniform(0.5, 2.0, ne)
    mask = rng.integers(0, 8, nn).astype(np.uint8)
    u = rng.standard_normal(3 * nn)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    E_d, m_d, u_d = dev(E), dev(mask), dev(u)
    y = torch.full((3 * nn,), float("nan"), dtype=torch.float64, device="cuda")
    dot = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    rc = _lib.load().vf_apply_noalloc(nx, ny, nz, 0.31, E_d.data_ptr(), m_d.data_ptr(), u_d.data_ptr(), y.data_ptr(),
                                      dot.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == _lib.VF_OK
    ke = torch.from_numpy(hex8.hex8_ke(1.0, 0.31)).cuda()
    edof = torch.from_numpy(hex8.build_edof(nx, ny, nz).astype(np.int64)).cuda()
    ref = torch.zeros_like(y).index_add_(0, edof.reshape(-1), ((u_d[edof] @ ke.T) * E_d[:, None]).reshape(-1))
    ref[((m_d[:, None].int() >> torch.arange(3, device="cuda")) & 1).reshape(-1) == 0] = 0.0
    scale = float(ref.abs().max())
    assert float((y - ref).abs().max()) <= 1e-13 * scale
    assert abs(dot.item() - float((u_d * ref).sum())) <= 1e-13 * float(u_d.abs().sum()) * scale
