"""The two kernel forms of 27-block Galerkin levels -- rows of nodes (FP64, and
FP32 up to 20,000 nodes) and the z-march (FP32 beyond) -- on both sides of that
limit and at ragged sizes.  The FP64 row form is checked against the sparse
oracle in test_gpu_ops.py; here the FP32 forms are compared with it.  A result
of either sums 81 products per component: FP32 storage rounds each value to
2^-24 (1e-6 of the largest result with the sum's own rounding), FP16 storage to
2^-11 (3e-3)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,rtol", [("sym_half", 3e-3), ("sym", 2e-6)])
@pytest.mark.parametrize("shape", [(2, 2, 2), (30, 14, 34), (52, 52, 52), (54, 52, 52), (66, 130, 20), (100, 54, 50)])
def test_level_forms(gpu, shape, storage, rtol):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = shape
    rng = np.random.default_rng(7)
    fixed = np.arange(3 * (nx + 1) * (ny + 1))
    m = MGSolver(nx, ny, nz, fixed, nu=0.3, min_elems=2, max_levels=2,
                 options=SolverOptions(coarse="galerkin", coarse_storage=storage))
    m.set_density(np.exp(rng.normal(0, 1, nx * ny * nz)))
    assert len(m.levels) == 2
    u = rng.standard_normal(m.levels[1]["ndof"])
    ref = m._apply(1, u, precision="fp64")
    got = m._apply(1, u, precision="fp32")
    scale = np.abs(ref).max()
    assert np.abs(got - ref).max() <= rtol * scale
    np.testing.assert_array_equal(got, m._apply(1, u, precision="fp32"))
    m.close()
