"""That the grids of the dissected coarsest solve's tests are dissected (three
kernels in a V-cycle where an explicit inverse is one; otherwise the launches of
a small grid of the same depth), and that the load cases of a block solve, which
share its blocks and run at the same time, each have their own vectors."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(dims, smoothed, levels):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = dims
    fixed = np.arange(3 * (nx + 1) * (ny + 1))
    m = MGSolver(nx, ny, nz, fixed, nu=0.3, n_smooth=0, max_levels=levels,
                 options=SolverOptions.robust(smoothed_transfers=smoothed, smoothed_level_sweeps=0, autotune=False))
    m.set_density(np.random.default_rng(0).uniform(0.5, 2.0, nx * ny * nz))
    return m


def _vcycle_launches(m, precision):
    from voxelsim_fea_b200 import _lib
    n = [ctypes.c_uint64(), ctypes.c_uint64()]
    b = np.ones(m.ndof)
    m._vcycle(0, b, precision=precision)
    _lib.check(_lib.load().vf_launch_count(ctypes.byref(n[0])), None)
    m._vcycle(0, b, precision=precision)
    _lib.check(_lib.load().vf_launch_count(ctypes.byref(n[1])), None)
    m.close()
    return n[1].value - n[0].value


@pytest.mark.parametrize("dims,smoothed,levels", [((72, 12, 8), 0, 2), ((8, 60, 12), 0, 2), ((12, 8, 66), 0, 2),
                                                  ((104, 16, 16), 2, 3), ((16, 88, 24), 2, 3), ((24, 16, 96), 2, 3)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_these_levels_are_dissected(gpu, dims, smoothed, levels, precision):
    small = (8, 8, 8) if levels == 2 else (16, 16, 16)
    assert _vcycle_launches(_solver(dims, smoothed, levels), precision) == \
        _vcycle_launches(_solver(small, smoothed, levels), precision) + 2


def test_block_cases_share_the_blocks_only(gpu):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = 72, 12, 8
    rng = np.random.default_rng(4)
    fixed = np.arange(3 * (nx + 1) * (ny + 1))
    E = rng.uniform(0.5, 2.0, nx * ny * nz)
    for options in (SolverOptions.robust(), SolverOptions.fast()):
        m = MGSolver(nx, ny, nz, fixed, nu=0.3, max_levels=2, options=options)
        F = rng.standard_normal((5, m.ndof))
        F[:, fixed] = 0.0
        U = m.solve_block(E, F, tol=1e-10)
        for f, u in zip(F, U):
            ref = m.solve(E, f, tol=1e-10)
            assert np.abs(u - ref).max() <= 1e-7 * np.abs(ref).max()
        m.close()
