"""The coarsest level's Jacobi sweeps from zero in one launch: a one-level
V-cycle is exactly those sweeps, compared with the oracle's V-cycle on grids at
the edges of its thread rounds (one element, fewer and more elements and nodes
than threads), one past what fits in shared memory (the sweeps launched one by
one), one and two sweeps, partly fixed nodes, a Poisson ratio per voxel, and
both precisions.  Tolerances: FP64 1e-12 of the largest value over 30
contractive sweeps, FP32 1e-4."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,sweeps", [((1, 1, 1), 30), ((16, 4, 4), 30), ((9, 7, 8), 30), ((8, 8, 8), 2),
                                         ((3, 5, 2), 1), ((11, 9, 7), 30), ((20, 10, 10), 30)])
@pytest.mark.parametrize("lame", [False, True])
def test_one_level_vcycle_is_the_sweeps(gpu, dims, sweeps, lame):
    from oracle import hex8
    from voxelsim_fea_b200 import _lib
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + sweeps)
    ne, ndof = nx * ny * nz, 3 * (nx + 1) * (ny + 1) * (nz + 1)
    E = rng.uniform(0.5, 2.0, ne)
    nu = rng.uniform(0.2, 0.4, ne) if lame else None
    fixed = np.unique(np.concatenate([np.arange(3 * (nx + 1)), rng.integers(0, ndof, 5)]))
    m = MGSolver(nx, ny, nz, fixed, nu=0.3, max_levels=1, omega=0.5,
                 options=SolverOptions(coarse_sweeps=sweeps, autotune=False))
    m.set_density(E, nu_elem=nu)
    edof = hex8.build_edof(nx, ny, nz)
    if lame:
        kl, km = np.empty(576), np.empty(576)
        _lib.check(_lib.load().vf_hex8_tables(0.3, None, _lib.ptr(kl), _lib.ptr(km), None))
        lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
        apply = lambda v: (hex8.element_apply(v, lam, edof, kl.reshape(24, 24), ndof)  # noqa: E731
                           + hex8.element_apply(v, mu, edof, km.reshape(24, 24), ndof))
    else:
        ke = hex8.hex8_ke(1.0, 0.3)
        apply = lambda v: hex8.element_apply(v, E, edof, ke, ndof)  # noqa: E731
    free = np.ones(ndof, bool)
    free[fixed] = False
    b = rng.standard_normal(ndof)
    minv = m.inv_diagonal(0)
    x = np.zeros(ndof)
    for _ in range(sweeps):
        x = x + np.where(free, 0.5 * minv * (b - np.where(free, apply(x), 0.0)), 0.0)
    scale = np.abs(x).max()
    assert np.abs(m._vcycle(0, b) - x).max() <= 1e-12 * scale
    assert np.abs(m._vcycle(0, b, precision="fp32") - x).max() <= 1e-4 * scale
    m.close()
