"""Algorithmic bytes that the persistent CG declares while profiling, for a system whose rows stay on chip: an
iteration does not count the matrix again.  Between a loose and a tight solve the declared bytes grow per iteration by
the vectors (17 Krylov and 3 V-cycle values per row of level 0, up to 8 of the coarse levels' rows, which are under
half of level 0's) and the dense coarsest matrix (at most 500 x 500), and by no less than 0.9 of the Krylov values.
A system of 512k cells streams its finest level: there an iteration counts its entries three times."""
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


@pytest.mark.parametrize("shape", [(24, 24, 24), (48, 48, 48), (80, 80, 80)], ids=lambda s: "x".join(map(str, s)))
def test_bytes_per_iteration(ctx, shape):
    import babelsim_b200 as bsg
    poly = meshgen.hex_box(*shape, flat=True)
    own, nbr = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64)
    inner, n = nbr >= 0, poly.n_cells
    rng = np.random.default_rng(5)
    c = np.where(inner, np.exp(0.3 * rng.standard_normal(len(own))), 0.0)
    d = np.full(n, 1e-3)
    np.add.at(d, own[inner], c[inner])
    np.add.at(d, nbr[inner], c[inner])
    b = rng.standard_normal(n)
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    system = bsg.LinearSystem(mesh)
    seen = []
    for rtol in (1e-3, 1e-3, 1e-5):
        ctx.profile(True)
        _, res = system.solve(bsg.solver_config("cg", "hypre", 1e-30, rtol, 500), d, -c, -c, b)
        _, _, declared, iterations = ctx.profile_report()["pcg_amg_persistent"]
        ctx.profile(False)
        assert res[0].status == 0
        seen.append((declared, iterations))
    (b0, i0), (b1, i1) = seen[1:]
    assert i1 > i0
    per = (b1 - b0) / (i1 - i0)
    if n < 200000:
        assert 0.9 * 17 * 8 * n <= per <= 24 * 8 * n + 8 * 500 * 500
    else:
        assert per >= 3 * 12 * 6 * n * 0.95
    system.close()
    mesh.close()
