"""A coarsest operator that is not positive definite is refused with the row of
the coarse operator (DOF 3 * node + component, x fastest) where a pivot failed,
whether the direct solve keeps one explicit inverse (the short grid) or dissects
the level: moduli of 1 and -0.99 in turn at one end (a positive diagonal that is
small beside the couplings across single coarse voxels) put that row at that
end.  Twice the same row."""

import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,axis", [((72, 12, 8), 0), ((8, 60, 12), 1), ((12, 8, 66), 2), ((12, 8, 4), 0)])
def test_reported_row_is_a_row_of_the_coarse_operator(gpu, dims, axis):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = dims
    ends = np.arange((nx + 1) * (ny + 1) * (nz + 1))
    coord = (ends % (nx + 1), ends // (nx + 1) % (ny + 1), ends // ((nx + 1) * (ny + 1)))[axis]
    fixed = (3 * ends[coord == 0][:, None] + np.arange(3)).ravel()
    cut = dims[axis] - 6
    ix = np.indices(dims)
    E = np.where((ix[axis] >= cut) & ((ix // 2).sum(axis=0) % 2 == 1), -0.99, 1.0)
    m = MGSolver(nx, ny, nz, fixed, nu=0.3, max_levels=2,
                 options=SolverOptions.robust(smoothed_transfers=0, smoothed_level_sweeps=0, autotune=False))
    rows = []
    for _ in range(2):
        with pytest.raises(RuntimeError, match="non-positive pivot") as err:
            m.set_density(E.ravel())
        rows.append(int(re.search(r"at row (\d+)", str(err.value)).group(1)))
    m.close()
    assert rows[0] == rows[1]
    c = [d // 2 + 1 for d in dims]
    node = rows[0] // 3
    at = (node % c[0], node // c[0] % c[1], node // (c[0] * c[1]))
    assert node < c[0] * c[1] * c[2] and at[axis] >= cut // 2, (rows, at)
