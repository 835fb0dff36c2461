"""The fine sweep with a Poisson ratio per voxel as a Chebyshev step (the previous
update loaded ahead of its use, three stages of the staging ring): a V-cycle with
the TMA-staged kernel is bit for bit that with the copy-staged one, chunked and in
one wave, on grids with several units per CTA, in both precisions; and on a small
grid it is the Chebyshev V-cycle restated with the solver's own level operators
(FP64, 1e-9 of the largest value: the coarse system's condition is below 1e6)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(dims):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    E = np.where(rng.random(nx * ny * nz) < 0.7, 1.0, 1e-2) * rng.uniform(0.5, 2.0, nx * ny * nz)
    nu = rng.uniform(0.2, 0.4, E.size)
    fixed = np.arange(3 * (nx + 1) * (ny + 1))
    b = rng.standard_normal(3 * (nx + 1) * (ny + 1) * (nz + 1))
    b[fixed] = 0.0
    return E, nu, fixed, b


def _solver(dims, fixed, **kw):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    return MGSolver(*dims, fixed, nu=0.3, max_levels=2,
                    options=SolverOptions.robust(smoothed_transfers=0, smoothed_level_sweeps=0, autotune=False, **kw))


@pytest.mark.parametrize("dims", [(64, 48, 40), (36, 30, 10), (120, 60, 52)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_staged_forms_are_bitwise_equal(gpu, dims, prec):
    E, nu, fixed, b = _problem(dims)
    out = []
    for kernel, zc in (("modal_cpasync", 5), ("modal", 3), ("modal", -1)):
        m = _solver(dims, fixed, fine_kernel=kernel, modal_zchunk=zc, coarsest="jacobi")
        m.set_density(E, nu_elem=nu)
        out.append(m._vcycle(0, b, precision=prec))
        m.close()
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 0
    np.testing.assert_array_equal(out[0], out[1])
    np.testing.assert_array_equal(out[1], out[2])


@pytest.mark.parametrize("zchunk", [3, -1])
def test_against_the_restated_vcycle(gpu, zchunk):
    dims = (14, 12, 8)
    E, nu, fixed, b = _problem(dims)
    m = _solver(dims, fixed, modal_zchunk=zchunk)
    m.set_density(E, nu_elem=nu)
    lam = m.level_omega(0)[1]
    theta, delta = 0.5 * (lam + lam / 30), 0.5 * (lam - lam / 30)
    rho0 = delta / theta
    rho1 = 1.0 / (2.0 / rho0 - rho0)
    minv = m.inv_diagonal(0)

    def smooth(x):
        d = minv * (b - m._apply(0, x)) / theta
        x = x + d
        return x + rho1 * rho0 * d + 2.0 * rho1 / delta * minv * (b - m._apply(0, x))

    x = smooth(np.zeros_like(b))
    rc = m._restrict(0, b - m._apply(0, x))
    A = np.empty((rc.size, rc.size))
    for j in range(rc.size):
        e = np.zeros(rc.size)
        e[j] = 1.0
        A[:, j] = m._apply(1, e)
    dead = np.diag(A) == 0
    A[dead, dead] = 1.0
    ref = smooth(x + m._prolongate(0, np.linalg.solve(A, rc)))
    assert np.abs(m._vcycle(0, b) - ref).max() <= 1e-9 * np.abs(ref).max()
    m.close()
