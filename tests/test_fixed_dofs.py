"""The fixed DOFs from the nodes' bits: the expansion of the supported nodes and
that of all nodes give the same list on both sides of the line between them."""

import numpy as np
import pytest


@pytest.mark.parametrize("share", [0.0, 0.01, 0.3, 0.36, 0.7, 1.0])
def test_both_expansions(share):
    from voxelsim_fea_b200.solve_worker import _fixed_dofs
    rng = np.random.default_rng(1)
    bits = np.where(rng.random(5000) < share, rng.integers(0, 8, 5000), 0).astype(np.uint8)
    if share == 1.0:
        bits[:] = 7
    flags = ((bits[:, None] >> np.arange(3)) & 1).astype(bool).ravel()
    ref = np.flatnonzero(flags)
    for count in (ref.size, 0, 3 * bits.size):   # (0 and all: either expansion whatever the bits)
        got = _fixed_dofs(bits, count)
        assert got.dtype == np.int64
        np.testing.assert_array_equal(got, ref)
