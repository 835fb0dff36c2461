"""What the autotuner's choice is kept by.  A solver's first set-up on a grid
times candidates (extra launches); the next on the same grid takes the choice
from the process's table.  A choice timed on one modulus must not serve two,
nor one precision the other, and a solver whose material changes kind takes the
choice of that kind.  Launch counts show which happened."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _count():
    from voxelsim_fea_b200 import _lib
    n = ctypes.c_uint64()
    _lib.check(_lib.load().vf_launch_count(ctypes.byref(n)), None)
    return n.value


def _setup(m, E, nu=None):
    a = _count()
    m.set_density(E, nu_elem=nu)
    return _count() - a


def test_one_choice_per_material_kind_and_precision(gpu):
    from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions
    nx, ny, nz = 40, 24, 36
    rng = np.random.default_rng(2)
    E = rng.uniform(0.5, 2.0, nx * ny * nz)
    nu = rng.uniform(0.2, 0.4, E.size)
    fixed = np.arange(3 * (nx + 1) * (ny + 1))
    new = lambda **kw: MGSolver(nx, ny, nz, fixed, nu=0.3, max_levels=1, options=SolverOptions(**kw))  # noqa: E731
    a = new()
    first, again = _setup(a, E), _setup(a, E)
    assert first > again                           # timed, then kept by the solver
    switched = _setup(a, E, nu)
    b = new()
    two = _setup(b, E, nu)
    assert switched > two                          # one modulus' choice did not serve two; two's own then did
    assert _setup(a, E) == again                   # back to one modulus: from the table
    c = new(precision="fp32")
    d = new(precision="fp32")
    assert _setup(c, E) > _setup(d, E)             # FP64's choice did not serve FP32
    for m in (a, b, c, d):
        m.close()
