"""GMRES with AMG pays for no structure that only the CG solvers read (tree numbering, folded coarse matrix):
its set-up issues the same launches with one smoothing step, for which CG has those structures, as with two,
for which there are none.  A zero right-hand side leaves nothing to iterate, so what is counted is the set-up
and a fixed rest.  CG after GMRES on the same system still gets its structures and meets the contract."""
import numpy as np
import pytest

from babelsim_b200 import meshgen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import babelsim_b200 as bsg
    c = bsg.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("ksp", ["gmres", "fgmres"])
@pytest.mark.parametrize("shape", [(6, 6, 6), (16, 16, 16), (26, 26, 26)], ids=lambda s: "x".join(map(str, s)))
def test_setup_launches(ctx, shape, ksp):
    import babelsim_b200 as bsg
    rng = np.random.default_rng([*shape])
    poly = meshgen.hex_box(*shape, flat=True)
    own, nbr = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64)
    inner, n = nbr >= 0, poly.n_cells
    c = np.where(inner, np.exp(0.3 * rng.standard_normal(len(own))), 0.0)
    d = np.full(n, 1e-2)
    np.add.at(d, own[inner], c[inner])
    np.add.at(d, nbr[inner], c[inner])
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    counts = {}
    for steps in (1, 2):
        system = bsg.LinearSystem(mesh)
        cfg = bsg.solver_config(ksp, "hypre", 1e-30, 1e-10, 500, amg_smoothing_steps=steps, rebuild_interval=1)
        counts[steps] = []
        for version in range(2):  # the structure, and a rebuild for new values
            before = ctx.launches()
            _, res = system.solve(cfg, d * (1.0 + version), -c, -c, np.zeros(n))
            assert res[0].status == 0
            counts[steps].append(ctx.launches() - before)
        if steps == 1:
            b = rng.standard_normal(n)
            x, res = system.solve(bsg.solver_config("cg", "hypre", 1e-30, 1e-10, 500), 2.0 * d, -c, -c, b)
            y = 2.0 * d * x
            np.add.at(y, own[inner], -c[inner] * x[nbr[inner]])
            np.add.at(y, nbr[inner], -c[inner] * x[own[inner]])
            assert res[0].status == 0 and np.linalg.norm(b - y) <= 1.01e-10 * np.linalg.norm(b)
        system.close()
    assert counts[1] == counts[2]
    mesh.close()
