"""Performance cases: the calls that programs built on this package spend their time in.

Every case goes through the Python API (the C ABI below it) as a solver loop, a serving process or a
drop-in linear-system backend does: one pass hands host arrays over (or continues on device-resident
state), lets the framework work, and takes whole fields back.

Sizes, boundary conditions, discretisations and solver controls are those of this repository's
benchmark, tests and serving loop.  Polyhedral meshes are jittered-lattice Voronoi cubes of
`meshgen.voronoi_cube`; the large ones are made of mirrored copies of a smaller cube, which meet face
to face, because the triangulation behind one large cube takes minutes.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

import babelsim_b200 as bsg
from babelsim_b200 import meshgen

MESH_SEED = 20261007
WALLS = 6
LID = 3


# ---------------------------------------------------------------- meshes
def _mirrored(base, m: int):
    """m^3 copies of a lattice-numbered Voronoi unit cube, odd copies mirrored per axis, as one mesh
    of the unit cube numbered along the whole lattice (x fastest)."""
    if m == 1:
        return base
    n = round(base.n_cells ** (1.0 / 3.0))
    off, ids = (np.asarray(a, np.int64) for a in base.flat())
    own, nbr, pat = (np.asarray(a, np.int64) for a in (base.owner, base.neighbour, base.patch))
    v, nv, sizes = np.asarray(base.vertices), len(base.vertices), np.diff(off)
    lat = np.stack([np.arange(n ** 3) % n, np.arange(n ** 3) // n % n, np.arange(n ** 3) // (n * n)], 1)
    face_of = np.repeat(np.arange(len(own)), sizes)
    on = np.zeros((nv, 6), bool)                     # vertices on each side of the cube
    for side in range(6):
        on[ids[pat[face_of] == side], side] = True
    interior, side_faces = np.nonzero(pat < 0)[0], [np.nonzero(pat == s)[0] for s in range(6)]

    def cells(b):
        g = [b[a] * n + (lat[:, a] if b[a] % 2 == 0 else n - 1 - lat[:, a]) for a in range(3)]
        return g[0] + m * n * (g[1] + m * n * g[2])

    def low_side(a, k):                              # the base side that faces copy k - 1 on axis a
        return 2 * a + (k % 2)
    rings, out_own, out_nbr, out_pat, out_sizes, verts = [], [], [], [], [], []
    for bz in range(m):
        for by in range(m):
            for bx in range(m):
                b = (bx, by, bz)
                cb = np.tile(np.array(b), (nv, 1))
                x = np.empty_like(v)
                for a in range(3):
                    # a vertex on a shared plane belongs to the lower of the two copies
                    if b[a] > 0:
                        cb[on[:, low_side(a, b[a])], a] -= 1
                    x[:, a] = (b[a] + (v[:, a] if b[a] % 2 == 0 else 1.0 - v[:, a])) / m
                key = (cb[:, 0] + m * (cb[:, 1] + m * cb[:, 2])) * nv + np.arange(nv)
                verts.append((key, x))
                c = cells(b)
                groups = [(interior, c[own[interior]], c[nbr[interior]], np.full(len(interior), -1))]
                for a in range(3):
                    lo, hi = low_side(a, b[a]), low_side(a, b[a]) ^ 1
                    if b[a] == 0:
                        f = side_faces[lo]
                        groups.append((f, c[own[f]], np.full(len(f), -1), np.full(len(f), 2 * a)))
                    f = side_faces[hi]
                    if b[a] == m - 1:
                        groups.append((f, c[own[f]], np.full(len(f), -1), np.full(len(f), 2 * a + 1)))
                    else:                            # meets its own mirror image in the next copy
                        nb = list(b)
                        nb[a] += 1
                        groups.append((f, c[own[f]], cells(nb)[own[f]], np.full(len(f), -1)))
                for f, o, nb_, p in groups:
                    s = sizes[f]
                    pos = np.repeat(off[f] - np.r_[0, np.cumsum(s)[:-1]], s) + np.arange(int(s.sum()))
                    rings.append(key[ids[pos]])
                    out_sizes.append(s)
                    flip = (nb_ >= 0) & (nb_ < o)
                    out_own.append(np.where(flip, nb_, o))
                    out_nbr.append(np.where(flip, o, nb_))
                    out_pat.append(p)
    key = np.concatenate([k for k, _ in verts])
    xyz = np.concatenate([x for _, x in verts])
    where = np.full(m ** 3 * nv, -1, np.int64)
    where[key[::-1]] = np.arange(len(key))[::-1]     # the first copy of each shared vertex
    kept = np.unique(where[where >= 0])
    new = np.full(len(key), -1, np.int64)
    new[kept] = np.arange(len(kept))
    flat = new[where[np.concatenate(rings)]]
    o, nb_, p, s = (np.concatenate(a) for a in (out_own, out_nbr, out_pat, out_sizes))
    order = np.lexsort((np.where(nb_ >= 0, nb_, 0), o, p))
    start = np.r_[0, np.cumsum(s)[:-1]][order]
    so = s[order]
    pos = np.repeat(start - np.r_[0, np.cumsum(so)[:-1]], so) + np.arange(int(so.sum()))
    i32 = np.int32
    return meshgen.PolyMesh(xyz[kept], None, o[order].astype(i32), nb_[order].astype(i32), p[order].astype(i32),
                            list(base.patch_names), list(base.patch_kinds),
                            offsets=np.r_[0, np.cumsum(so)].astype(i32), ids=flat[pos].astype(i32))


@lru_cache(maxsize=6)
def _poly(n: int, m: int):
    return _mirrored(meshgen.voronoi_cube(n, 0.3, MESH_SEED), m)


@lru_cache(maxsize=6)
def _hex(nx: int, ny: int, nz: int, lx: float, ly: float, lz: float):
    return meshgen.hex_box(nx, ny, nz, (0.0, 0.0, 0.0), (lx, ly, lz), flat=True)


@lru_cache(maxsize=1)
def _context():
    return bsg.Context(0)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _swirl(x, rng, speed, axes=3):
    """A divergence-free cellular flow along the first `axes` axes that does not cross the box's walls,
    and a smooth pressure."""
    lo, ext = x.min(0), np.maximum(np.ptp(x, axis=0), 1e-12)
    s = np.pi * (x - lo) / ext
    U, p = np.zeros_like(x), np.zeros(len(x))
    for _ in range(4):
        a, b = rng.choice(axes, 2, replace=False)
        ka, kb = rng.integers(1, 4, 2)
        amp = speed * rng.uniform(-0.3, 0.3)
        U[:, a] += amp * np.sin(ka * s[:, a]) * np.cos(kb * s[:, b])
        U[:, b] -= amp * (ka * ext[b]) / (kb * ext[a]) * np.cos(ka * s[:, a]) * np.sin(kb * s[:, b])
        p += speed * rng.uniform(-0.1, 0.1) * np.cos(ka * s[:, a]) * np.cos(kb * s[:, b])
    return U, p


class _State:
    """What a program keeps between calls; closes its device objects when it is dropped."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        kept = self.__dict__
        for o in [kept.get("eq"), kept.get("system"), kept.get("sim"), *kept.get("fields", []), kept.get("mesh")]:
            if o is not None:
                o.close()


# ---------------------------------------------------------------- the cases
def _poly_case(name, n, m, **kw):
    return {**({"name": name} if name else {}), "kind": "simple", "mesh": "poly", "n": n, "m": m, "p_precision": 0,
            "u_precision": 0, "nu": 1e-3, **kw}


def listed():
    return [
        # the tests' 12 x 12 cavity: the smallest solve, all launches, host steps and barriers
        {"name": "cavity-144", "kind": "simple", "mesh": "cavity", "n": 12, "nu": 0.01},
        # the 64 x 64 cavity of the reference's own case directory
        {"name": "cavity-4096", "kind": "simple", "mesh": "cavity", "n": 64, "nu": 0.01},
        # a serving-sized polyhedral cavity with the benchmark's methods
        _poly_case("poly-33k", 32, 1),
        # the mixed-precision options (FP32 V-cycle, FP32 inner momentum solve) on the benchmark's 48^3 sample size
        _poly_case("poly-110k-mixed", 24, 2, p_precision=2, u_precision=1),
        # the benchmark's one-million-cell polyhedral cavity, one outer iteration with host copies
        _poly_case("poly-1m", 25, 4),
        # eight uneven cavities advanced as one block-diagonal batch (the serving loop's cohort)
        {"name": "batch-8", "kind": "batch", "cases": "v16 v20 v24 v28 v32 v40 h20 h32"},
        # transient PISO past a cylinder, one time step of the 200k-cell O-grid
        {"name": "piso-200k", "kind": "piso", "n_theta": 2000, "n_r": 100, "dt": 0.001},
        # steady RANS: SIMPLE + k-omega in a tanh-stretched plane channel
        {"name": "komega-1m", "kind": "komega", "nx": 160, "ny": 100, "nz": 64},
        # a new case from its mesh to its fields: ingest, set-up (AMG structure included), ten outer iterations
        {"name": "job-14k", "kind": "job", "n": 24, "iterations": 10},
        # the drop-in linear-system seam: a pressure-like system with new values on every call
        {"name": "system-cg-64k", "kind": "system", "mesh": "poly", "n": 20, "m": 2, "components": 1, "ksp": "cg",
         "pc": "hypre"},
        # the seam's momentum system: three right-hand sides, one non-symmetric matrix
        {"name": "system-bcgs3-97k", "kind": "system", "mesh": "hex", "n": 46, "m": 1, "components": 3,
         "ksp": "bcgs", "pc": "bjacobi"},
        # an implicit transport step assembled with the equation API
        {"name": "transport-295k", "kind": "transport", "nx": 96, "ny": 64, "nz": 48, "dt": 0.01, "gamma": 1e-3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cavity", "poly", "poly", "mixed", "batch", "piso", "komega", "job", "system", "system",
                       "transport"])
    if kind == "cavity":
        return {"kind": "simple", "mesh": "cavity", "n": _log(rng, 12, 200), "nu": rng.choice([0.01, 0.005])}
    if kind in ("poly", "mixed"):
        m = rng.choice([1, 2, 3, 4] if kind == "poly" else [1, 2, 3])
        over = {} if kind == "poly" else {"p_precision": 2, "u_precision": rng.choice([0, 1])}
        return _poly_case(None, _log(rng, 9, 24), m, nu=round(math.exp(rng.uniform(math.log(1e-3), math.log(1e-2))), 6),
                          **over)
    if kind == "batch":
        return {"kind": "batch", "cases": " ".join(rng.choice("vh") + str(rng.randint(12, 30))
                                                   for _ in range(rng.randint(2, 10)))}
    if kind == "piso":
        return {"kind": "piso", "n_theta": _log(rng, 200, 2000), "n_r": _log(rng, 40, 100), "dt": 0.001}
    if kind == "komega":
        return {"kind": "komega", "nx": _log(rng, 16, 160), "ny": _log(rng, 24, 100), "nz": _log(rng, 8, 64)}
    if kind == "job":
        return {"kind": "job", "n": rng.randint(12, 28), "iterations": rng.randint(5, 15)}
    if kind == "system":
        mesh = rng.choice(["poly", "hex"])
        ksp, pc, comps = rng.choice([("cg", "hypre", 1), ("cg", "jacobi", 1), ("bcgs", "bjacobi", 3),
                                     ("bcgs", "bjacobi", 1), ("gmres", "hypre", 1), ("fgmres", "hypre", 1)])
        return {"kind": "system", "mesh": mesh, "n": _log(rng, 12, 24 if mesh == "poly" else 64),
                "m": rng.choice([1, 2]) if mesh == "poly" else 1, "components": comps, "ksp": ksp, "pc": pc}
    return {"kind": "transport", "nx": _log(rng, 17, 120), "ny": _log(rng, 17, 80), "nz": _log(rng, 5, 48),
            "dt": rng.choice([0.01, 0.05]), "gamma": rng.choice([1e-3, 1e-2])}


# ---------------------------------------------------------------- SIMPLE, single case
def _benchmark_simple(mesh, nu, p_precision=0, u_precision=0):
    o = bsg.options("linear", "leastSquares", "linearUpwind", "corrected")
    return bsg.Simple(mesh, 1.0, nu, 0.7, 0.3, 2, 1e-8, 1e-7, 1e-6, 1e-6, o, o,
                      bsg.solver_config("bcgs", "bjacobi", 1e-14, 1e-10, 1000, precision=u_precision),
                      bsg.solver_config("cg", "hypre", 1e-14, 1e-10, 1000, precision=p_precision))


def _lid(sim, patch0, speed):
    for k in range(WALLS):
        sim.set_boundary("U", patch0 + k, "fixedValue", (speed, 0.0, 0.0) if k == LID else (0.0, 0.0, 0.0))
        sim.set_boundary("p", patch0 + k, "zeroGradient")


def _resident(mesh, sim, U, p):
    """Fields set, and the pinned host arrays that each pass copies in and out."""
    sim.set_fields(U, p)
    s = _State(mesh=mesh, sim=sim, U=_pinned(U.shape), p=_pinned(p.shape), phi=_pinned((mesh.n_faces,)),
               out=[_pinned(U.shape), _pinned(p.shape), _pinned((mesh.n_faces,))])
    s.U[:], s.p[:] = U, p
    s.phi[:] = sim.fields()[2]
    return s


def _prepare_simple(case, rng):
    if case["mesh"] == "cavity":
        poly = _cavity(case["n"])
        mesh = bsg.Mesh.from_polyhedral(_context(), poly)
        sim = bsg.Simple(mesh, 1.0, case["nu"], 0.7, 0.3, 1, 1e-6, 1e-6, 1e-6, 1e-6, bsg.options(), bsg.options(),
                         bsg.solver_config("bcgs", "bjacobi", 1e-15, 1e-10, 2000),
                         bsg.solver_config("cg", "hypre", 1e-15, 1e-10, 5000))
        speed = rng.uniform(0.5, 2.0)
        for k in range(6):
            wall = k < 4
            sim.set_boundary("U", k, "fixedValue" if wall else "symmetry", (speed if k == 3 else 0.0, 0.0, 0.0))
            sim.set_boundary("p", k, "zeroGradient" if wall else "symmetry")
    else:
        mesh = bsg.Mesh.from_polyhedral(_context(), _poly(case["n"], case["m"]))
        sim = _benchmark_simple(mesh, case["nu"], case["p_precision"], case["u_precision"])
        speed = rng.uniform(0.5, 2.0)
        _lid(sim, 0, speed)
    U, p = _swirl(mesh.export("cell_centres"), rng, speed, 2 if case["mesh"] == "cavity" else 3)
    return _resident(mesh, sim, U, p)


@lru_cache(maxsize=8)
def _cavity(n):
    return meshgen.cavity_2d(n)


def _run_resident(s):
    s.sim.load_state(s.U, s.p, s.phi)
    s.sim.iterate(1)
    s.sim.fields_into(*s.out)
    return {"U": s.out[0], "p": s.out[1], "phi": s.out[2]}


# ---------------------------------------------------------------- batch
def _batch_meshes(text):
    return [_poly(int(t[1:]), 1) if t[0] == "v" else _hex(int(t[1:]), int(t[1:]), int(t[1:]), 1.0, 1.0, 1.0)
            for t in text.split()]


def _prepare_batch(case, rng):
    poly, cells, patches = _batch_poly(case["cases"])
    k = len(cells) - 1
    nu = np.exp(rng.uniform(np.log(1e-3), np.log(1e-2), k))
    mesh = bsg.Mesh.from_polyhedral(_context(), poly)
    sim = _benchmark_simple(mesh, float(nu[0]))
    sim.set_segments(cells, nu)
    x = mesh.export("cell_centres")
    U, p = np.zeros((mesh.n_cells, 3)), np.zeros(mesh.n_cells)
    for q in range(k):
        a, b = int(cells[q]), int(cells[q + 1])
        speed = rng.uniform(0.5, 2.0)
        _lid(sim, int(patches[q]), speed)
        U[a:b], p[a:b] = _swirl(x[a:b], rng, speed)
    return _resident(mesh, sim, U, p)


@lru_cache(maxsize=4)
def _batch_poly(text):
    return meshgen.concatenate(_batch_meshes(text))


# ---------------------------------------------------------------- PISO
@lru_cache(maxsize=2)
def _ogrid(n_theta, n_r):
    return meshgen.cylinder_ogrid(n_theta, n_r, 0.5, 15.0, 1.05)


def _prepare_piso(case, rng):
    mesh = bsg.Mesh.from_polyhedral(_context(), _ogrid(case["n_theta"], case["n_r"]))
    o = bsg.options("linear", "leastSquares", "linearUpwind", "corrected")
    sim = bsg.Piso(mesh, 1.0, 0.01, 1.0, 1, 2, None, None, 1, 1e-7, 1e-7, 1e-6, 1e-7, "bdf2", 0.0, 1e9, case["dt"],
                   o, o, bsg.solver_config("bcgs", "bjacobi", 1e-15, 1e-12, 1000),
                   bsg.solver_config("cg", "hypre", 1e-15, 1e-12, 1500))
    speed = rng.uniform(0.8, 1.2)
    for k, (kind, v) in enumerate([("fixedValue", (0, 0, 0)), ("fixedValue", (speed, 0, 0)), ("zeroGradient", 0),
                                   ("symmetry", 0), ("symmetry", 0)]):
        sim.set_boundary("U", k, kind, v)
    for k, kind in enumerate(["zeroGradient", "zeroGradient", "fixedValue", "symmetry", "symmetry"]):
        sim.set_boundary("p", k, kind, 0.0)
    x = mesh.export("cell_centres")
    # potential flow past the cylinder, with a seeded circulation
    r2, g = x[:, 0] ** 2 + x[:, 1] ** 2, rng.uniform(-0.2, 0.2)
    U = np.zeros((mesh.n_cells, 3))
    U[:, 0] = speed * (1.0 - 0.25 * (x[:, 0] ** 2 - x[:, 1] ** 2) / r2 ** 2) - g * x[:, 1] / r2
    U[:, 1] = speed * (-0.5 * x[:, 0] * x[:, 1] / r2 ** 2) + g * x[:, 0] / r2
    sim.set_fields(U, np.zeros(mesh.n_cells))
    return _State(mesh=mesh, sim=sim)


def _run_piso(s):
    s.sim.advance(1)
    U, p, phi = s.sim.fields()
    return {"U": U, "p": p, "phi": phi}


# ---------------------------------------------------------------- k-omega channel
@lru_cache(maxsize=2)
def _channel(nx, ny, nz):
    return meshgen.channel(nx, ny, nz)


def _prepare_komega(case, rng):
    mesh = bsg.Mesh.from_polyhedral(_context(), _channel(case["nx"], case["ny"], case["nz"]))
    o = bsg.options("linear", "greenGauss", "linearUpwind", "orthogonal")
    t = bsg.options("linear", "greenGauss", "upwind", "orthogonal")
    sim = bsg.Simple(mesh, 1.0, 1e-4, 0.7, 0.3, 0, 1e-8, 1e-7, 1e-6, 1e-6, o, o,
                     bsg.solver_config("bcgs", "bjacobi", 1e-14, 1e-10, 1000),
                     bsg.solver_config("cg", "hypre", 1e-14, 1e-10, 1000))
    sim.enable_komega(k_transport=t, omega_transport=t, k_solver=bsg.solver_config("bcgs", "bjacobi", 1e-18, 1e-12, 1000),
                      omega_solver=bsg.solver_config("bcgs", "bjacobi", 1e-18, 1e-12, 1000))
    speed, k0 = rng.uniform(0.8, 1.2), 3.75e-3 * rng.uniform(0.5, 2.0)
    for name, bcs in (("U", [(speed, 0, 0), None, (0, 0, 0), (0, 0, 0)]), ("p", [None, 0.0, None, None]),
                      ("k", [k0, None, 1e-12, 1e-12]), ("omega", [10.0, None, 1e4, 1e4])):
        for patch, v in enumerate(bcs):
            sim.set_boundary(name, patch, "zeroGradient" if v is None else "fixedValue", 0.0 if v is None else v)
        for patch in (4, 5):
            sim.set_boundary(name, patch, "symmetry")
    x = mesh.export("cell_centres")
    n = mesh.n_cells
    y = np.minimum(x[:, 1], 2.0 - x[:, 1])
    k = k0 * (1.0 - np.exp(-40.0 * y)) + 1e-12
    omega = 10.0 + 50.0 / (y + 0.01)
    sim.set_turbulence_fields(k, omega)
    U = np.zeros((n, 3))
    U[:, 0] = speed * (1.0 - (1.0 - y) ** 8)
    s = _resident(mesh, sim, U, np.zeros(n))
    s.k, s.omega = k, omega
    return s


def _run_komega(s):
    s.sim.set_turbulence_fields(s.k, s.omega)
    out = _run_resident(s)
    out["k"], out["omega"], out["mut"] = s.sim.turbulence_fields()
    return out


# ---------------------------------------------------------------- a whole job
def _prepare_job(case, rng):
    return _State(poly=_poly(case["n"], 1), speed=rng.uniform(0.5, 2.0),
                  nu=float(np.exp(rng.uniform(np.log(1e-3), np.log(1e-2)))), iterations=case["iterations"])


def _run_job(s):
    mesh = bsg.Mesh.from_polyhedral(_context(), s.poly)
    sim = _benchmark_simple(mesh, s.nu)
    _lid(sim, 0, s.speed)
    sim.set_fields(np.zeros((mesh.n_cells, 3)), np.zeros(mesh.n_cells))
    sim.iterate(s.iterations)
    U, p, phi = sim.fields()
    sim.close()
    mesh.close()
    return {"U": U, "p": p, "phi": phi}


# ---------------------------------------------------------------- the linear-system seam
def _system_mesh(case):
    return _poly(case["n"], case["m"]) if case["mesh"] == "poly" else _hex(case["n"], case["n"], case["n"], 1.0, 1.0, 1.0)


def _system_arrays(case, seed):
    """Two versions of a diffusion(-convection) matrix in the caller's face order, and a right-hand side."""
    rng = np.random.default_rng(seed)
    poly = _system_mesh(case)
    own, nbr = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64)
    inner, n = nbr >= 0, poly.n_cells
    h = 1.0 / round(n ** (1.0 / 3.0))
    symmetric = case["ksp"] == "cg" or case["pc"] == "hypre"
    versions = []
    for _ in range(2):
        c = h * np.exp(0.3 * rng.standard_normal(len(own)))
        flux = np.zeros(len(own)) if symmetric else h * rng.standard_normal(len(own))
        up = np.where(inner, -c + np.minimum(flux, 0.0), 0.0)
        lo = np.where(inner, -c - np.maximum(flux, 0.0), 0.0)
        d = np.zeros(n)
        np.add.at(d, own[inner], -up[inner])
        np.add.at(d, nbr[inner], -lo[inner])
        fixed = ~inner & (np.asarray(poly.patch) == 1) if symmetric else ~inner
        np.add.at(d, own[fixed], 2.0 * c[fixed])
        if not symmetric:                            # a relaxed or transient term
            d *= 1.2
        versions.append((d, up, lo))
    b = rng.standard_normal((n, 3) if case["components"] == 3 else n)
    return versions, b


def _prepare_system(case, seed):
    versions, b = _system_arrays(case, seed)
    mesh = bsg.Mesh.from_polyhedral(_context(), _system_mesh(case))
    return _State(mesh=mesh, system=bsg.LinearSystem(mesh, case["components"]), versions=versions, b=b, turn=0,
                  cfg=bsg.solver_config(case["ksp"], case["pc"], 1e-30, 1e-12, 3000))


def _run_system(s):
    d, up, lo = s.versions[s.turn]
    s.turn ^= 1
    x, _ = s.system.solve(s.cfg, d, up, lo, s.b)
    return x


def _exact_solution(product, diag, b):
    """BiCGStab with Jacobi to the last bits, restarted on the true residual (torch, FP64)."""
    x = torch.zeros_like(b)
    best, best_norm = x, math.inf
    for _ in range(8):
        r = b - product(x)
        norm = float(torch.linalg.norm(r))
        if norm < best_norm:
            best, best_norm = x.clone(), norm
        if norm <= 2e-15 * float(torch.linalg.norm(b)):
            break
        r0, p = r.clone(), r.clone()
        rho = torch.dot(r0, r)
        for it in range(4000):
            ph = p / diag
            v = product(ph)
            alpha = rho / torch.dot(r0, v)
            s = r - alpha * v
            sh = s / diag
            t = product(sh)
            omega = torch.dot(t, s) / torch.dot(t, t)
            x = x + alpha * ph + omega * sh
            r = s - omega * t
            if it % 8 == 0 and not float(torch.linalg.norm(r)) > 1e-9 * norm:
                break
            new = torch.dot(r0, r)
            p = r + (new / rho) * (alpha / omega) * (p - omega * v)
            rho = new
    return best


def _exact_system(case, seed):
    versions, b = _system_arrays(case, seed)
    poly = _system_mesh(case)
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")

    def put(a, dtype=torch.float64):
        return torch.as_tensor(np.ascontiguousarray(a)).to(device, dtype)
    inner = np.asarray(poly.neighbour) >= 0
    own, nbr = put(poly.owner[inner], torch.int64), put(poly.neighbour[inner], torch.int64)
    d, up, lo = (put(a if len(a) == poly.n_cells else a[inner]) for a in versions[0])

    def product(x):
        return (d * x).index_add_(0, own, up * x[nbr]).index_add_(0, nbr, lo * x[own])
    cols = [_exact_solution(product, d, put(b if b.ndim == 1 else b[:, c])) for c in range(case["components"])]
    return (cols[0] if b.ndim == 1 else torch.stack(cols, 1)).cpu().numpy()


# ---------------------------------------------------------------- implicit transport, equation API
def _transport_box(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return nx, ny, nz, nx / 64.0, ny / 64.0, nz / 64.0


def _transport_inputs(case, rng):
    nx, ny, nz, *_ = _transport_box(case)
    x = np.stack(np.meshgrid(np.arange(nz) / nz, np.arange(ny) / ny, np.arange(nx) / nx, indexing="ij"), -1).reshape(-1, 3)
    old = 1.0 + 0.5 * np.sin(2 * np.pi * (x @ rng.integers(1, 4, 3))) + 0.05 * rng.standard_normal(len(x))
    return old, rng.standard_normal(len(x)), rng.uniform(0.5, 2.0), rng.uniform(0.5, 1.5)


def _prepare_transport(case, rng):
    poly = _hex(*_transport_box(case))
    old, source, speed, inlet = _transport_inputs(case, rng)
    mesh = bsg.Mesh.from_polyhedral(_context(), poly)
    o = bsg.options("linear", "greenGauss", "upwind", "orthogonal")
    x = bsg.Field(mesh, "cell", 1)
    x.set_boundary(0, "fixedValue", inlet)
    for k in range(1, 6):
        x.set_boundary(k, "zeroGradient")
    previous, src = bsg.Field(mesh, "cell", 1, old), bsg.Field(mesh, "cell", 1, source)
    velocity = bsg.Field(mesh, "cell", 3, np.tile([speed, 0.0, 0.0], (mesh.n_cells, 1)))
    velocity.set_boundary(0, "fixedValue", (speed, 0.0, 0.0))
    for k in range(1, 6):
        velocity.set_boundary(k, "zeroGradient" if k == 1 else "symmetry")
    phi = bsg.flux(velocity, o)
    return _State(mesh=mesh, eq=bsg.Equation(x, o), x=x, previous=previous, source=src, phi=phi,
                  fields=[x, previous, src, velocity, phi], dt=case["dt"], gamma=case["gamma"],
                  cfg=bsg.solver_config("bcgs", "bjacobi", 1e-30, 1e-12, 2000))


def _run_transport(s):
    s.eq.reset()
    s.eq.ddt(1.0, s.previous, s.dt)
    s.eq.div(s.phi)
    s.eq.laplacian(s.gamma, -1.0)
    s.eq.source(s.source)
    s.eq.solve(s.cfg)
    return s.x.download()


def _exact_transport(case, rng):
    nx, ny, nz, lx, ly, lz = _transport_box(case)
    old, source, speed, inlet = _transport_inputs(case, rng)
    h = (lx / nx, ly / ny, lz / nz)
    V = h[0] * h[1] * h[2]
    area = (h[1] * h[2], h[0] * h[2], h[0] * h[1])
    g = [case["gamma"] * area[a] / h[a] for a in range(3)]
    F = speed * area[0]
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    diag = torch.full((nz, ny, nx), V / case["dt"], dtype=torch.float64, device=device)
    b = torch.as_tensor((V / case["dt"]) * old + V * source).to(device).reshape(nz, ny, nx).clone()
    diag[:, :, 1:] += g[0]
    diag[:, :, :-1] += g[0]
    diag[:, 1:] += g[1]
    diag[:, :-1] += g[1]
    diag[1:] += g[2]
    diag[:-1] += g[2]
    diag += F                                        # every cell sends F downstream, the last one out of the box
    diag[:, :, 0] += 2.0 * g[0]
    b[:, :, 0] += (2.0 * g[0] + F) * inlet

    def product(flat):
        x = flat.reshape(nz, ny, nx)
        y = diag * x
        y[:, :, 1:] -= (g[0] + F) * x[:, :, :-1]
        y[:, :, :-1] -= g[0] * x[:, :, 1:]
        y[:, 1:] -= g[1] * x[:, :-1]
        y[:, :-1] -= g[1] * x[:, 1:]
        y[1:] -= g[2] * x[:-1]
        y[:-1] -= g[2] * x[1:]
        return y.reshape(-1)
    return _exact_solution(product, diag.reshape(-1), b.reshape(-1)).cpu().numpy()


# ---------------------------------------------------------------- dispatch
_PREPARE = {"simple": _prepare_simple, "batch": _prepare_batch, "piso": _prepare_piso, "komega": _prepare_komega,
            "job": _prepare_job, "transport": _prepare_transport}
_RUN = {"simple": _run_resident, "batch": _run_resident, "piso": _run_piso, "komega": _run_komega, "job": _run_job,
        "transport": _run_transport, "system": _run_system}


def prepare(case, seed):
    kind = case["kind"]
    s = _prepare_system(case, seed) if kind == "system" else _PREPARE[kind](case, np.random.default_rng(seed))
    s.kind = kind
    return s


def run(state):
    return _RUN[state.kind](state)


def exact(case, seed):
    if case["kind"] == "system":
        return _exact_system(case, seed)
    if case["kind"] == "transport":
        return _exact_transport(case, np.random.default_rng(seed))
    return None                                      # an outer iteration has no short plain form


def _size(case):
    """(cells, faces), estimated from the generators' numbers."""
    kind = case["kind"]
    if kind == "transport":
        return _box_size(case["nx"], case["ny"], case["nz"])
    if kind == "komega":
        return _box_size(case["nx"], case["ny"], case["nz"])
    if kind == "piso":
        n = case["n_theta"] * case["n_r"]
        return n, 4 * n
    if kind == "job":
        return case["n"] ** 3, 7.7 * case["n"] ** 3
    if kind == "batch":
        sizes = [(int(t[1:]) ** 3, (7.7 if t[0] == "v" else 3.1) * int(t[1:]) ** 3) for t in case["cases"].split()]
        return sum(c for c, _ in sizes), sum(f for _, f in sizes)
    if case["mesh"] == "cavity":
        return case["n"] ** 2, 4 * case["n"] ** 2
    n = (case["n"] * case.get("m", 1)) ** 3
    return n, (7.7 if case["mesh"] == "poly" else 3.1) * n


def _box_size(nx, ny, nz):
    return nx * ny * nz, 3 * nx * ny * nz + nx * ny + ny * nz + nx * nz


def work(case):
    """Each input array read once and each result written once (FP64 8 B, indices 4 B); one multiply and
    one add per matrix entry for each system that a pass solves.  Krylov iterations are not counted: how
    many there are is the method's choice."""
    cells, faces = _size(case)
    kind = case["kind"]
    mesh = 40.0 * cells + 152.0 * faces
    entry = 2.0 * (cells + 2.0 * faces)
    if kind == "system":
        c = case["components"]
        return {"bytes": 8.0 * cells * (1 + 2 * c) + 16.0 * faces + 8.0 * faces, "flops": entry * c}
    if kind == "transport":
        return {"bytes": 48.0 * cells + 40.0 * faces, "flops": entry}
    passes = case["iterations"] if kind == "job" else 1
    systems = 3 + {"piso": 4, "komega": 3}.get(kind, 1 if case.get("mesh") == "cavity" else 3)
    fields = 2.0 * (32.0 * cells + 8.0 * faces) + (40.0 * cells if kind == "komega" else 0.0)
    return {"bytes": mesh + fields, "flops": passes * systems * entry}
