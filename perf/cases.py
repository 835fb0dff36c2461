"""Performance cases: what a user of this framework has it compute, through its
public entry points, from the smallest call to the largest.

Kinds of case
  matvec     vf_apply_noalloc: y = K u and u.y on the caller's device buffers
             (the operator by itself, FP64), for programs with their own solver
  reference  MGSolver with its defaults (the FP64 algorithm with rediscretized
             levels and 30 Jacobi sweeps on the coarsest) on a solid cantilever
  job        VoxelFEA as a solve job uses it: solve, von Mises stress, mean
             displacement per voxel; the fields in FP32, as a job delivers them.
             Grids that cannot be coarsened enough (most odd sizes) take its
             Jacobi-PCG, the others its multigrid, "fp64" (its default) or "mixed"
  solve      MGSolver with the mixed-precision preset on a large or two-material
             part, page-locked arrays in and out, converged to where the FP64
             displacement itself is the result
  block      MGSolver.solve_block: several load cases on one part
  batch      solve_batch: independent parts of uneven sizes in one call
  voxelize   the voxel phase of a job: inside tests of the part, support and load
             meshes, grid assembly, island removal
  conv       one 3x3x3 convolution of the learned stage, forward and backward

Parts are the package's seeded noise parts (void voxels at 1e-9 of the modulus)
after the island step that every job passes through, with a load on a random top
patch of what is left.
"""

import math

import numpy as np
import torch

from voxelsim_fea_b200 import _lib, generators, inside, solve_worker
from voxelsim_fea_b200.fea import VoxelFEA
from voxelsim_fea_b200.learned import conv
from voxelsim_fea_b200.multigrid import MGSolver, SolverOptions, solve_batch

E_MIN = 1e-9
DENSE_MAX = 16384        # DOFs of the coarsest level that the direct solve takes
CONV_PAIRS = ((16, 16), (16, 32), (32, 16), (32, 32), (32, 64), (64, 32), (64, 64))


def listed():
    return [
        # the operator on a small grid: an outer loop of the caller's own, where the call itself counts
        {"name": "matvec 48x24x24", "kind": "matvec", "nx": 48, "ny": 24, "nz": 24},
        # the operator on an odd grid of millions of nodes: bandwidth
        {"name": "matvec 251x127x129", "kind": "matvec", "nx": 251, "ny": 127, "nz": 129},
        # the reference algorithm on its own demonstration beam: a few milliseconds of small launches
        {"name": "reference 64x16x16", "kind": "reference", "nx": 64, "ny": 16, "nz": 16, "levels": 3, "tol": 1e-8},
        # an interactive job on a coarse grid with the mixed-precision preset
        {"name": "job mixed 64x32x32", "kind": "job", "nx": 64, "ny": 32, "nz": 32, "precision": "mixed"},
        # a job whose grid is odd in every direction: Jacobi-PCG, thousands of short iterations
        {"name": "job odd 61x43x37", "kind": "job", "nx": 61, "ny": 43, "nz": 37, "precision": "fp64"},
        # a job whose grid coarsens only twice: a coarsest level of 10,920 DOFs to factor
        {"name": "job fp64 100x52x36", "kind": "job", "nx": 100, "ny": 52, "nz": 36, "precision": "fp64"},
        # an ordinary job with the job worker's own settings
        {"name": "job fp64 128x64x64", "kind": "job", "nx": 128, "ny": 64, "nz": 64, "precision": "fp64"},
        # two materials (a Poisson ratio per voxel): a few hundred iterations on a middling grid
        {"name": "solve two-material 96x80x64", "kind": "solve", "nx": 96, "ny": 80, "nz": 64, "materials": 2,
         "tol": 1e-11},
        # the large bracket of the benchmark
        {"name": "solve bracket 256x128x128", "kind": "solve", "nx": 256, "ny": 128, "nz": 128, "materials": 1,
         "tol": 1e-11},
        # a batch of uneven parts: many small solves at once
        {"name": "batch of 6 parts", "kind": "batch",
         "shapes": "32x48x64,64x64x64,96x32x48,48x80x32,112x64x48,64x32x96"},
        # the voxel phase of a job with a part mesh of ten thousand triangles
        {"name": "voxelize 128x96x64", "kind": "voxelize", "nx": 128, "ny": 96, "nz": 64, "triangles": 10000},
        # a training step's unit: one layer of the network on the box of a level-1 node grid
        {"name": "conv 32-32 68x52x36", "kind": "conv", "x": 68, "y": 52, "z": 36, "cin": 32, "cout": 32},
    ]


# -- sizes -----------------------------------------------------------------------------------------


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _coarsest_dofs(dims, max_levels=6, min_elems=4):
    """DOFs of the coarsest level of the multigrid hierarchy on a grid."""
    d, n = list(dims), 1
    while n < max_levels and all(v % 2 == 0 for v in d) and min(d) // 2 >= min_elems // 2:
        d = [v // 2 for v in d]
        n += 1
    return 3 * (d[0] + 1) * (d[1] + 1) * (d[2] + 1)


def draw(rng):
    kind = rng.choice(("matvec", "reference", "job", "job", "solve", "block", "batch", "voxelize", "conv"))
    if kind == "matvec":
        # 3,000 to 4 million nodes, every residue
        n = math.exp(rng.uniform(math.log(3e3), math.log(4e6)))
        a, b = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
        s = n ** (1.0 / 3.0)
        return {"kind": kind, "nx": max(4, int(s * a)), "ny": max(4, int(s * b)), "nz": max(4, int(s / (a * b)))}
    if kind == "reference":
        # beams up to three times as long as thick: its rediscretized levels lose most slenderer ones
        ny, nz = 4 * rng.randint(3, 8), 4 * rng.randint(3, 8)
        nx = 4 * rng.randint(4, min(16, 3 * min(ny, nz) // 4))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "levels": rng.choice((2, 3, 4)), "tol": 1e-8}
    if kind == "job":
        while True:
            nx, ny, nz = (_log_int(rng, 20, 140) for _ in range(3))
            if rng.random() < 0.6:      # a user who asks for a round size
                nx, ny, nz = (max(24, v // 8 * 8) for v in (nx, ny, nz))
            multigrid = _coarsest_dofs((nx, ny, nz)) <= DENSE_MAX
            if nx * ny * nz <= (1_000_000 if multigrid else 120_000):
                return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": rng.choice(("fp64", "mixed"))}
    if kind in ("solve", "block"):
        while True:
            nx, ny, nz = (8 * _log_int(rng, 5, 28) for _ in range(3))
            if _coarsest_dofs((nx, ny, nz)) > 9000:
                continue
            if kind == "solve" and 200_000 <= nx * ny * nz <= 700_000:
                return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "materials": rng.choice((1, 2)), "tol": 1e-11}
            if kind == "block" and nx * ny * nz <= 300_000:
                return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "cases": rng.randint(2, 6)}
    if kind == "batch":
        n = rng.randint(2, 8)
        edges = (32, 48, 64, 80, 96)
        return {"kind": kind, "shapes": ",".join("%dx%dx%d" % tuple(rng.choice(edges) for _ in range(3))
                                                 for _ in range(n))}
    if kind == "voxelize":
        while True:
            nx, ny, nz = (_log_int(rng, 24, 160) for _ in range(3))
            t = _log_int(rng, 200, 40000)
            if nx * ny * nz * t <= 8e9:
                return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "triangles": t}
    cin, cout = rng.choice(CONV_PAIRS)
    x, y, z = (4 * _log_int(rng, 4, 25) for _ in range(3))
    return {"kind": "conv", "x": x, "y": y, "z": z, "cin": cin, "cout": cout}


# -- inputs ----------------------------------------------------------------------------------------


def _part(shape, seed, materials=1):
    """A seeded part after the island step, with what of it is active, its supports and one load."""
    for k in range(32):
        s = seed + 100_003 * k
        make = generators.bracket if materials == 1 else generators.two_material_part
        p = generators.drop_unsupported(make(tuple(shape), seed=s % (1 << 31), sigma=3.0 if min(shape) < 48 else 4.0))
        solid = p["active"].mean()
        if p["fixed_dofs"].size and solid > 0.2:
            break
    p["f"] = generators.load_cases(p, 1, seed + 1)[0]
    p["E"] = np.where(p["active"], p["E_stiff"], p["E_stiff"] * E_MIN)
    return p


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _torus(triangles, size, rng):
    """A closed, bumpy torus that fills a box of `size`, of about so many triangles."""
    nv = max(6, int(math.sqrt(triangles / 6.0)))
    nu = max(8, int(triangles / (2 * nv)))
    a = np.linspace(0.0, 2.0 * np.pi, nu, endpoint=False)[:, None]
    b = np.linspace(0.0, 2.0 * np.pi, nv, endpoint=False)[None, :]
    bump = 1.0 + 0.15 * np.sin(rng.integers(2, 6) * a + rng.uniform(0, 6)) * np.cos(rng.integers(1, 4) * b)
    r = 0.14 * bump
    x, y, z = (0.32 + r * np.cos(b)) * np.cos(a), (0.32 + r * np.cos(b)) * np.sin(a), 2.2 * r * np.sin(b) + 0 * a
    verts = (np.stack([x, y, z], axis=-1).reshape(-1, 3) + 0.5) * np.asarray(size)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    v = lambda di, dj: (((i + di) % nu) * nv + (j + dj) % nv).ravel()  # noqa: E731
    faces = np.concatenate([np.stack([v(0, 0), v(1, 0), v(1, 1)], 1), np.stack([v(0, 0), v(1, 1), v(0, 1)], 1)])
    return verts, faces.astype(np.int64)


def _box(lo, hi):
    lo, hi = np.asarray(lo, dtype=float), np.asarray(hi, dtype=float)
    verts = np.array([[(lo, hi)[(k >> c) & 1][c] for c in range(3)] for k in range(8)])
    quads = [(0, 2, 3, 1), (4, 5, 7, 6), (0, 1, 5, 4), (2, 6, 7, 3), (0, 4, 6, 2), (1, 3, 7, 5)]
    faces = [t for q in quads for t in ((q[0], q[1], q[2]), (q[0], q[2], q[3]))]
    return verts, np.asarray(faces, dtype=np.int64)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    dims = tuple(case[k] for k in ("nx", "ny", "nz")) if "nx" in case else None
    s = {"kind": kind, "case": case}
    if kind == "matvec":
        ne, nn = dims[0] * dims[1] * dims[2], (dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1)
        g = torch.Generator(device="cuda").manual_seed(seed)
        solid = torch.rand(ne, generator=g, device="cuda") < 0.5
        s["E"] = torch.where(solid, 69e6, 69e6 * E_MIN).double()
        s["mask"] = torch.full((nn,), 7, dtype=torch.uint8, device="cuda")
        s["mask"][:(dims[0] + 1) * (dims[1] + 1)] = 0            # the z = 0 face is clamped
        s["u"] = torch.randn(3 * nn, generator=g, device="cuda", dtype=torch.float64)
        s["y"], s["dot"] = torch.empty_like(s["u"]), torch.empty(1, dtype=torch.float64, device="cuda")
        return s
    if kind == "reference":
        p = generators.cantilever(*dims, load_n=float(rng.uniform(500.0, 1500.0)))
        face = p["f"].reshape(-1, 3)[:, 2:] != 0                  # the loaded end: bent across the beam
        s["f"] = (face * np.append(0.0, rng.normal(0.0, 1.0, 2)) * abs(p["f"].min())).ravel()
        s["E"] = p["E_stiff"] * float(rng.uniform(0.5, 1.5))
        s["solver"] = MGSolver(*dims, p["fixed_dofs"], nu=p["nu"], max_levels=case["levels"])
        return s
    if kind == "job":
        p = _part(dims, seed)
        opt = SolverOptions.fast() if case["precision"] == "mixed" else None
        fea = VoxelFEA(*dims, nu=p["nu"], active_elems=p["active"].reshape(dims), mg_options=opt)
        fea.set_fixed(p["fixed_dofs"])
        s.update(fea=fea, E=p["E_stiff"], E_stress=p["E_stress"], f=p["f"], vsize=p["vsize"], dims=dims)
        return s
    if kind == "solve":
        p = _part(dims, seed, case["materials"])
        two = case["materials"] == 2
        s["solver"] = MGSolver(*dims, p["fixed_dofs"], nu=0.3 if two else p["nu"], options=SolverOptions.fast())
        s["E"], s["f"], s["out"] = _pinned(p["E"]), _pinned(p["f"]), _pinned(np.zeros(p["f"].size))
        s["nu"] = _pinned(p["nu"]) if two else None
        return s
    if kind == "block":
        p = _part(dims, seed)
        s["solver"] = MGSolver(*dims, p["fixed_dofs"], nu=p["nu"], options=SolverOptions.fast())
        s["E"], s["F"] = p["E"], generators.load_cases(p, case["cases"], seed + 1)
        return s
    if kind == "batch":
        parts = [_part([int(v) for v in t.split("x")], seed + 31 * i)
                 for i, t in enumerate(case["shapes"].split(","))]
        s["solvers"] = [MGSolver(*p["dims"], p["fixed_dofs"], nu=p["nu"], options=SolverOptions.fast())
                        for p in parts]
        s["E"], s["F"] = [p["E"] for p in parts], [p["f"] for p in parts]
        return s
    if kind == "voxelize":
        vs = 1e-3
        size = np.asarray(dims) * vs
        cut = float(rng.uniform(0.15, 0.25))
        s.update(dims=dims, vsize=vs, origin=np.zeros(3), part=_torus(case["triangles"], size, rng),
                 support=_box((-vs, -vs, -vs), (size[0] * cut, size[1] + vs, size[2] + vs)),
                 load=_box((size[0] * (1.0 - cut), -vs, -vs), size + vs),
                 force=tuple(float(v) for v in rng.normal(0.0, 500.0, 3)))
        return s
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["z"], case["y"], case["x"])
    new = lambda *d: torch.randn(*d, generator=g, device="cuda")  # noqa: E731
    s["x"] = torch.relu(new(*shape, case["cin"])).bfloat16().requires_grad_()
    s["w"] = (new(27, case["cout"], case["cin"]) * math.sqrt(2.0 / (27 * case["cin"]))).requires_grad_()
    s["b"] = (0.1 * new(case["cout"])).requires_grad_()
    s["dy"] = new(*shape, case["cout"]).bfloat16()
    return s


# -- one pass --------------------------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind == "matvec":
        c = s["case"]
        rc = _lib.load().vf_apply_noalloc(c["nx"], c["ny"], c["nz"], 0.33, s["E"].data_ptr(), s["mask"].data_ptr(),
                                          s["u"].data_ptr(), s["y"].data_ptr(), s["dot"].data_ptr(),
                                          torch.cuda.current_stream().cuda_stream)
        _lib.check(rc, None, "matvec")
        return s["y"], s["dot"]
    if kind == "reference":
        return s["solver"].solve(s["E"], s["f"], tol=s["case"]["tol"])
    if kind == "job":
        u = s["fea"].solve(s["E"], s["f"], tol=1e-8)
        vm = s["fea"].element_von_mises_stress(u, s["E_stress"]) / s["vsize"]
        return {"stress": vm.astype(np.float32), "displacement": solve_worker.element_displacement(u, s["dims"])}
    if kind == "solve":
        return s["solver"].solve(s["E"], s["f"], tol=s["case"]["tol"], nu_elem=s["nu"], out=s["out"])
    if kind == "block":
        U = s["solver"].solve_block(s["E"], s["F"], tol=1e-8)
        return [solve_worker.element_displacement(u, (s["solver"].nx, s["solver"].ny, s["solver"].nz)) for u in U]
    if kind == "batch":
        U = solve_batch(s["solvers"], s["E"], s["F"], tol=1e-8)
        return [solve_worker.element_displacement(u, (m.nx, m.ny, m.nz)) for m, u in zip(s["solvers"], U)]
    if kind == "voxelize":
        grid = (s["dims"], s["origin"], s["vsize"])
        masks = [inside.inside_grid(*s["part"], *grid, "centers"), inside.inside_grid(*s["support"], *grid, "nodes"),
                 inside.inside_grid(*s["load"], *grid, "nodes")]
        descr = [("build", None), ("bearing", (1, 1, 1)), ("load", s["force"])]
        active, _, force, bits = solve_worker.assemble(descr, masks, s["dims"])
        kept, removed = solve_worker.drop_unsupported_islands_bits(active, bits, s["dims"])
        return {"kept": kept, "bits": bits, "force": force, "removed": removed}
    s["x"].grad = s["w"].grad = s["b"].grad = None
    y = conv.conv3d(s["x"], s["w"], s["b"])
    y.backward(s["dy"])
    return {"y": y.detach(), "dx": s["x"].grad, "dw": s["w"].grad, "db": s["b"].grad}


# -- work and 64-bit results -----------------------------------------------------------------------


def work(case):
    """Inputs read once, results written once; the operator's modal form takes about 170 operations a voxel."""
    kind = case["kind"]
    if kind == "conv":
        v = case["x"] * case["y"] * case["z"]
        return {"bytes": v * (4 * case["cin"] + 4 * case["cout"]) + 27 * 8 * case["cin"] * case["cout"],
                "flops": 3 * 2 * 27 * v * case["cin"] * case["cout"]}
    if kind == "batch":
        all_dims = [[int(v) for v in t.split("x")] for t in case["shapes"].split(",")]
    else:
        all_dims = [[case["nx"], case["ny"], case["nz"]]]
    ne = sum(a * b * c for a, b, c in all_dims)
    nn = sum((a + 1) * (b + 1) * (c + 1) for a, b, c in all_dims)
    if kind == "matvec":
        return {"bytes": 8 * ne + nn + 48 * nn, "flops": 170 * ne}
    if kind == "voxelize":
        return {"bytes": 60 * case["triangles"] + 2 * ne + 2 * nn + 25 * nn, "flops": 40 * ne}
    k = case.get("cases", 1)
    # a solve cannot do with less than one application of the operator for each decimal digit
    digits = -math.log10(case.get("tol", 1e-8))
    return {"bytes": 8 * ne * case.get("materials", 1) + 48 * nn * k, "flops": 170 * ne * digits * k}


def _ke(nu):
    """24x24 stiffness of the unit hexahedron, unit modulus, 2x2x2 Gauss points (x fastest, then y, then z corners)."""
    c = 1.0 / ((1 + nu) * (1 - 2 * nu))
    C = np.diag([1 - nu] * 3 + [(1 - 2 * nu) / 2] * 3) * c
    C[:3, :3] += nu * c * (1 - np.eye(3))
    corners = np.array([[(k >> a) & 1 for a in range(3)] for k in range(8)])
    K = np.zeros((24, 24))
    for gp in range(8):
        x = 0.5 + (2 * corners[gp] - 1) / (2 * math.sqrt(3.0))
        n1 = np.where(corners == 1, x, 1 - x)
        d = np.stack([(2 * corners[:, a] - 1) * np.prod(np.delete(n1, a, 1), 1) for a in range(3)], 1)
        B = np.zeros((6, 24))
        for a in range(3):
            B[a, a::3] = d[:, a]
        for r, (a, b) in enumerate(((0, 1), (1, 2), (2, 0))):
            B[3 + r, a::3], B[3 + r, b::3] = d[:, b], d[:, a]
        K += B.T @ C @ B / 8
    return K


def _operator(dims, E, nu):
    """u (z, y, x, 3) -> K u in torch, 64 bits; E in element order iz-fastest."""
    nx, ny, nz = dims
    K = torch.as_tensor(_ke(nu), device="cuda")
    Ez = E.reshape(nx, ny, nz).permute(2, 1, 0).unsqueeze(-1)
    cut = [(slice(k >> 2, nz + (k >> 2)), slice((k >> 1) & 1, ny + ((k >> 1) & 1)), slice(k & 1, nx + (k & 1)))
           for k in range(8)]

    def apply(u):
        q = (torch.cat([u[c] for c in cut], dim=-1) @ K) * Ez
        y = torch.zeros_like(u)
        for k, c in enumerate(cut):
            y[c] += q[..., 3 * k:3 * k + 3]
        return y
    return apply, Ez, torch.diagonal(K).reshape(8, 3), cut


def _cg(dims, E, nu, free, f, most=20000, tol=1e-13):
    """Jacobi-preconditioned CG in torch, 64 bits."""
    apply, Ez, dk, cut = _operator(dims, E, nu)
    d = torch.zeros_like(f)
    for k, c in enumerate(cut):
        d[c] += Ez * dk[k]
    minv = torch.where(free, 1.0 / d, torch.zeros_like(d))
    f = torch.where(free, f, torch.zeros_like(f))
    u, r = torch.zeros_like(f), f.clone()
    z = minv * r
    p, rz, stop = z.clone(), (r * z).sum(), (tol * f.norm()) ** 2
    for it in range(most):
        q = torch.where(free, apply(p), torch.zeros_like(p))
        a = rz / (p * q).sum()
        u += a * p
        r -= a * q
        z = minv * r
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
        if it % 50 == 49 and float((r * r).sum()) < float(stop):
            break
    return u


def exact(case, seed):
    kind = case["kind"]
    if kind == "conv":
        s = prepare(case, seed)
        x, w, b = (t.detach().double().requires_grad_() for t in (s["x"], s["w"].detach().bfloat16(), s["b"]))
        k = w.permute(1, 2, 0).reshape(case["cout"], case["cin"], 3, 3, 3)
        xp = torch.nn.functional.pad(x.permute(3, 0, 1, 2), (1, 1, 1, 1, 1, 1))
        Z, Y, X = case["z"], case["y"], case["x"]
        y = b.expand(Z, Y, X, -1)
        for t in range(27):
            a = xp[:, t // 9:t // 9 + Z, t // 3 % 3:t // 3 % 3 + Y, t % 3:t % 3 + X].permute(1, 2, 3, 0)
            y = y + a @ k[:, :, t // 9, t // 3 % 3, t % 3].T
        y.backward(s["dy"].double())
        return {"y": y.detach(), "dx": x.grad, "dw": w.grad, "db": b.grad}
    if kind == "matvec":
        s = prepare(case, seed)
        dims = (case["nx"], case["ny"], case["nz"])
        shape = (dims[2] + 1, dims[1] + 1, dims[0] + 1, 3)
        y = _operator(dims, s["E"], 0.33)[0](s["u"].reshape(shape))
        y[s["mask"].reshape(shape[:3]) == 0] = 0.0
        y = y.reshape(-1)
        return y, (s["u"] * y).sum().reshape(1)
    if kind not in ("reference", "job") or case["nx"] * case["ny"] * case["nz"] > 200_000:
        return None
    dims = (case["nx"], case["ny"], case["nz"])
    shape = (dims[2] + 1, dims[1] + 1, dims[0] + 1, 3)
    s = prepare(case, seed)
    dev = lambda a: torch.as_tensor(np.asarray(a), device="cuda")  # noqa: E731
    free = torch.ones(shape, dtype=torch.bool, device="cuda")
    if kind == "reference":
        free.reshape(-1)[dev(s["solver"]._fixed)] = False
        u = _cg(dims, dev(s["E"]), 0.3, free, dev(s["f"]).reshape(shape))
        return u.reshape(-1)
    fea = s["fea"]
    multigrid = _coarsest_dofs(dims) <= DENSE_MAX       # the Jacobi-PCG leaves the void voxels out
    act = dev(fea.active_elems)
    E = dev(s["E"]) * torch.where(act, 1.0, E_MIN if multigrid else 0.0).double()
    free.reshape(-1)[dev(fea._fixed_dofs_full)] = False
    if not multigrid:
        used = torch.zeros(free.numel(), dtype=torch.bool, device="cuda")
        used[dev(fea.used_dofs)] = True
        free &= used.reshape(shape)
    u = _cg(dims, E, fea.nu, free, dev(s["f"]).reshape(shape))
    nu = fea.nu
    c = 1.0 / ((1 + nu) * (1 - 2 * nu))
    nx, ny, nz = dims
    corner = [u[k >> 2:nz + (k >> 2), (k >> 1) & 1:ny + ((k >> 1) & 1), k & 1:nx + (k & 1)] for k in range(8)]
    disp = sum(v.norm(dim=-1) for v in corner) / 8
    g = [sum((1 if (k >> a) & 1 else -1) * corner[k] for k in range(8)) / 4 for a in range(3)]   # du/dx_a at the centre
    e = [g[a][..., a] for a in range(3)]
    tr = nu * (e[0] + e[1] + e[2])
    sg = [c * ((1 - 2 * nu) * v + tr) for v in e]
    ta = [c * (1 - 2 * nu) / 2 * (g[b][..., a] + g[a][..., b]) for a, b in ((0, 1), (1, 2), (2, 0))]
    vm = (0.5 * ((sg[0] - sg[1]) ** 2 + (sg[1] - sg[2]) ** 2 + (sg[2] - sg[0]) ** 2)
          + 3 * (ta[0] ** 2 + ta[1] ** 2 + ta[2] ** 2)).sqrt()
    order = lambda t: t.permute(2, 1, 0).reshape(-1)  # noqa: E731
    vm = torch.where(act, order(vm) * dev(s["E_stress"]) / s["vsize"], torch.zeros_like(order(vm)))
    return {"stress": vm, "displacement": order(disp)}
