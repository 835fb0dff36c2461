"""The dissected coarsest solve (interiors, separators as thick as the
stencil's reach) on coarsest levels long along each axis, at both reaches, with
fixed DOFs inside, several parts, and right where a part is one plane thicker
than another.  With no smoothing a V-cycle is P A_c^-1 P^T r, so it is compared
with the device's own transfers around a host FP64 solve with A_c taken from
the device column by column.  Tolerances: FP64 1e-9 of the largest value (the
condition of A_c is below 1e6 here), FP32 blocks 1e-3."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((72, 12, 8), 0, 2), ((8, 60, 12), 0, 2), ((12, 8, 66), 0, 2), ((104, 16, 16), 2, 3), ((16, 88, 24), 2, 3),
         ((24, 16, 96), 2, 3)]


@pytest.mark.parametrize("dims,smoothed,levels", CASES)
def test_vcycle_without_smoothing_is_the_coarse_solve(gpu, dims, smoothed, levels):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    E = np.where(rng.random(nx * ny * nz) < 0.6, 1.0, 0.05)
    nn = (nx + 1) * (ny + 1) * (nz + 1)
    ends = np.arange(nn)
    axis = int(np.argmax(dims))
    coord = (ends % (nx + 1), ends // (nx + 1) % (ny + 1), ends // ((nx + 1) * (ny + 1)))[axis]
    fixed = (3 * ends[(coord == 0) | (coord == dims[axis])][:, None] + np.arange(3)).ravel()
    fixed = np.concatenate([fixed, 3 * ends[coord == dims[axis] // 2][:7] + 1])
    m = MGSolver(nx, ny, nz, np.unique(fixed), nu=0.3, n_smooth=0, max_levels=levels,
                 options=SolverOptions.robust(smoothed_transfers=smoothed, smoothed_level_sweeps=0, autotune=False))
    m.set_density(E)
    lc = levels - 1
    assert len(m.levels) == levels
    n = m.levels[lc]["ndof"]
    A = np.empty((n, n))
    for j in range(n):
        e = np.zeros(n)
        e[j] = 1.0
        A[:, j] = m._apply(lc, e)
    dead = np.abs(np.diag(A)) == 0
    A[dead, dead] = 1.0
    r = rng.standard_normal(m.ndof)
    r[fixed] = 0.0
    b = r
    for li in range(lc):
        b = m._restrict(li, b)
    z = np.linalg.solve(A, b)
    for li in reversed(range(lc)):
        z = m._prolongate(li, z)
    scale = np.abs(z).max()
    assert np.abs(m._vcycle(0, r) - z).max() <= 1e-9 * scale
    assert np.abs(m._vcycle(0, r, precision="fp32") - z).max() <= 1e-3 * scale
    m.close()
