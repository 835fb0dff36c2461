"""The grid form of the inside test (each triangle visits only the grid points
its projection along the ray can cover) against the general form on the same
points given explicitly: equal masks, bit for bit, over ray directions with
each dominant axis and sign, both targets, flat and odd grids, meshes of a few
large and of many small triangles, open meshes of random slivers (edge-on
triangles, whose barycentric rounding is largest), far-away origins, and
vertices on grid planes.  And the tiled island fill against the oracle's
flood fill on a winding channel that crosses many tiles."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIRS = (None, (-1.0, 0.02, 0.5), (0.3, 1.0, -0.2), (0.1, -2.0, 0.3), (0.0, 0.0, 1.0), (0.01, 0.9, -1.0),
        (1.0, 1.0, 1.0))


def _mesh(kind, size, rng):
    if kind == "box":
        lo, hi = 0.2 * size, 0.8 * size
        v = np.array([[(lo, hi)[(k >> c) & 1][c] for c in range(3)] for k in range(8)])
        q = [(0, 2, 3, 1), (4, 5, 7, 6), (0, 1, 5, 4), (2, 6, 7, 3), (0, 4, 6, 2), (1, 3, 7, 5)]
        f = [t for a in q for t in ((a[0], a[1], a[2]), (a[0], a[2], a[3]))]
        return v, np.array(f)
    if kind == "slivers":   # random triangles, half of them nearly edge-on or degenerate
        n = 400
        c = rng.uniform(-0.1, 1.1, (n, 1, 3)) * size
        v = c + rng.normal(0, 0.1, (n, 3, 3)) * size
        v[::2, 2] = 0.5 * (v[::2, 0] + v[::2, 1]) + rng.normal(0, 1e-7, (n // 2, 3)) * size
        v[::8, 1] = v[::8, 0]
        return v.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3)
    nu, nv = 40, 24         # bumpy torus
    a = np.linspace(0, 2 * np.pi, nu, endpoint=False)[:, None]
    b = np.linspace(0, 2 * np.pi, nv, endpoint=False)[None, :]
    r = 0.15 * (1 + 0.2 * np.sin(3 * a))
    p = np.stack([(0.3 + r * np.cos(b)) * np.cos(a), (0.3 + r * np.cos(b)) * np.sin(a), 2 * r * np.sin(b) + 0 * a], -1)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    at = lambda di, dj: (((i + di) % nu) * nv + (j + dj) % nv).ravel()  # noqa: E731
    f = np.concatenate([np.stack([at(0, 0), at(1, 0), at(1, 1)], 1), np.stack([at(0, 0), at(1, 1), at(0, 1)], 1)])
    return (p.reshape(-1, 3) + 0.5) * size, f


@pytest.mark.parametrize("dims,vs,origin", [((17, 23, 9), 1e-3, (0, 0, 0)), ((1, 40, 3), 0.25, (5.0, -7.0, 1e3)),
                                            ((33, 8, 31), 2.0, (-30.0, 1e4, 0.5))])
@pytest.mark.parametrize("kind", ["box", "slivers", "torus"])
def test_grid_form_equals_point_form(gpu, kind, dims, vs, origin):
    from voxelsim_fea_b200 import inside
    rng = np.random.default_rng(11)
    size = np.asarray(dims) * vs
    v, f = _mesh(kind, size, rng)
    v = v + np.asarray(origin, dtype=float)
    for d in DIRS:
        d = None if d is None else np.asarray(d) / np.linalg.norm(d)
        for target, pts in (("centers", inside.voxel_centers(dims, origin, vs)),
                            ("nodes", inside.node_coords(dims, origin, vs))):
            np.testing.assert_array_equal(inside.inside_grid(v, f, dims, origin, vs, target, d),
                                          inside.inside_mask(v, f, pts, d), err_msg=f"{kind} {dims} {d} {target}")


def test_island_fill_across_tiles(gpu):
    from oracle import islands
    from voxelsim_fea_b200 import fea
    nx, ny, nz = 21, 19, 70
    act = np.zeros((nx, ny, nz), dtype=bool)
    for k, x in enumerate(range(0, nx, 2)):            # a channel that winds through every second x-plane
        for m, y in enumerate(range(0, ny, 2)):
            act[x, y, :] = True
            if y + 2 < ny:
                act[x, y + 1, -1 if m % 2 == 0 else 0] = True
        if x + 2 < nx:
            act[x + 1, ny - 1 if k % 2 == 0 else 0, 3] = True
    act[5, 5, 40] = True                               # an island
    fixed = np.array([0, 1, 2])
    kept, removed = fea.drop_unsupported_islands(act, fixed)
    ref, ref_removed = islands.drop_unsupported_islands(act, fixed)
    np.testing.assert_array_equal(kept, ref)
    assert removed == ref_removed
