"""The coarsest level's Jacobi sweeps run the operator kernel that the caller
chose: with "gather" or "modal_cpasync" a one-level V-cycle is bit for bit the
same number of smoothing sweeps from zero with that kernel (the first one, b - A 0,
is exact), in both precisions."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["gather", "modal_cpasync"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_coarsest_sweeps_use_the_chosen_kernel(gpu, kernel, precision):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = 9, 7, 8
    rng = np.random.default_rng(5)
    fixed = np.arange(3 * (nx + 1))
    m = MGSolver(nx, ny, nz, fixed, nu=0.3, max_levels=1, omega=0.5,
                 options=SolverOptions(coarse_sweeps=30, autotune=False, fine_kernel=kernel))
    m.set_density(rng.uniform(0.5, 2.0, nx * ny * nz))
    b = rng.standard_normal(m.ndof)
    b[fixed] = 0.0
    z = m._vcycle(0, b, precision=precision)
    x = m._smooth(0, np.zeros(m.ndof), b, 30, precision=precision)
    assert np.abs(x).max() > 0
    np.testing.assert_array_equal(z, x)
    m.close()
