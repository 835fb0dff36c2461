"""vf_apply_noalloc where its two forms and their tiles end: one-voxel grids,
exact tiles and one node past them, thin grids on both sides of the rule that
picks the gather form, many z-chunks and single planes, several calls in a row
(the ring of completion counters wraps) -- against a plain FP64 evaluation of
sum_e E_e Ke u_e.  Tolerance: 8 elements x 24 products per value, 1e-13 of the
result's largest value as for the other FP64 operators."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = ((1, 1, 1), (30, 6, 1), (31, 7, 2), (30, 6, 40), (61, 13, 5), (62, 14, 3), (5, 4, 3), (2, 70, 9), (70, 2, 9),
        (3, 41, 50), (1, 1, 400), (64, 20, 33))


@pytest.mark.parametrize("dims", DIMS)
def test_forms_against_plain_sum(gpu, dims):
    import torch
    from oracle import hex8
    from voxelsim_fea_b200 import _lib
    nx, ny, nz = dims
    nu = 0.31
    rng = np.random.default_rng(sum(dims))
    nn, ne = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    E = np.where(rng.random(ne) < 0.5, 1.0, 1e-9) * rng.uniform(0.5, 2.0, ne)
    mask = rng.integers(0, 8, nn).astype(np.uint8)
    free = ((mask[:, None] >> np.arange(3)) & 1).astype(bool).ravel()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    E_d, m_d = dev(E), dev(mask)
    y, dot = torch.empty(3 * nn, dtype=torch.float64, device="cuda"), torch.empty(1, dtype=torch.float64, device="cuda")
    edof, ke = hex8.build_edof(nx, ny, nz), hex8.hex8_ke(1.0, nu)
    for call in range(3):
        u = rng.standard_normal(3 * nn)
        u_d = dev(u)
        for _ in range(40):
            y.fill_(float("nan"))
            dot.fill_(float("nan"))
            rc = _lib.load().vf_apply_noalloc(nx, ny, nz, nu, E_d.data_ptr(), m_d.data_ptr(), u_d.data_ptr(),
                                              y.data_ptr(), dot.data_ptr(), torch.cuda.current_stream().cuda_stream)
            assert rc == _lib.VF_OK
        ref = hex8.element_apply(u, E, edof, ke, 3 * nn) * free
        scale = max(np.abs(ref).max(), 1e-300)
        assert np.abs(y.cpu().numpy() - ref).max() <= 1e-13 * scale
        assert abs(dot.item() - float(u @ ref)) <= 1e-13 * np.abs(u).sum() * scale
