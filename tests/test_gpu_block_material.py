"""The load cases of a block solve follow a change of the material's kind: the
launch graphs that the cases keep hold the operator of one modulus or of two."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_block_cases_follow_the_material_kind(gpu):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = 24, 16, 16
    rng = np.random.default_rng(3)
    E = rng.uniform(0.5, 2.0, nx * ny * nz)
    nu = rng.uniform(0.1, 0.4, E.size)
    fixed = np.arange(3 * (nx + 1) * (ny + 1))
    m = MGSolver(nx, ny, nz, fixed, nu=0.3, options=SolverOptions.robust())
    F = rng.standard_normal((3, m.ndof))
    F[:, fixed] = 0.0
    m.solve_block(E, F, tol=1e-10)
    for kind in (nu, None):
        U = m.solve_block(E, F, tol=1e-10, nu_elem=kind)
        for k in range(3):
            u = m.solve(E, F[k], tol=1e-10, nu_elem=kind)
            assert np.abs(U[k] - u).max() <= 1e-7 * np.abs(u).max()
    m.close()
