"""The displacement of a two-material solve stays what it was.  At a residual
of 1e-11 the nodes inside the void (1e-9 of the modulus) are not determined to
1e-9, so there the result follows the rounding of the FP32 V-cycle through
hundreds of iterations: the order of the level operators' sums, of the power
iteration that sets their damping, and of the first r.z.  The golden values
(4,000 DOFs of a 96x80x64 part, 395 iterations) were taken with one launch per
power step and norm, block by block row sums and full-grid reductions; 1e-9 of
their norm and 4e-8 of the largest are allowed.  (The autotuner is off: its
split groups the sums of p.Ap.)"""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "two_material_96x80x64.npz")


def test_two_material_displacement(gpu):
    from voxelsim_fea_b200 import generators
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    g = np.load(GOLDEN)
    dims = (96, 80, 64)
    p = generators.drop_unsupported(generators.two_material_part(dims, seed=4, sigma=4.0))
    f = generators.load_cases(p, 1, 5)[0]
    E = np.where(p["active"], p["E_stiff"], 1e-9 * p["E_stiff"])
    np.testing.assert_allclose([E.sum(), f.sum(), np.abs(f).sum(), p["nu"].sum()], g["checks"], rtol=1e-12)
    m = MGSolver(*dims, p["fixed_dofs"], nu=0.3, options=SolverOptions.fast(autotune=False))
    u = m.solve(E, f, tol=1e-11, nu_elem=p["nu"])
    at = np.unique(np.random.default_rng(0).integers(0, u.size, 4000))
    d = u[at] - g["u"]
    assert np.linalg.norm(d) <= 1e-9 * np.linalg.norm(g["u"])
    assert np.abs(d).max() <= 4e-8 * float(g["largest"])
    m.close()
