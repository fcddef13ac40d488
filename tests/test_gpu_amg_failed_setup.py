"""An AMG set-up that fails leaves nothing behind: the same call again is refused again, and a system that
can be coarsened is solved afterwards.

More than 2048 rows that nothing couples cannot be coarsened to a dense matrix, so coarsening stalls.  The
residual bound is the solver's contract with 1 % for the recomputation's own rounding."""
import numpy as np
import pytest

from babelsim_b200 import meshgen

pytestmark = pytest.mark.gpu
RTOL = 1e-10


@pytest.fixture(scope="module")
def ctx():
    import babelsim_b200 as bsg
    c = bsg.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("solver,precision", [("cg", 0), ("cg", 1), ("cg", 2), ("gmres", 0)])
@pytest.mark.parametrize("cut", [1.0, 0.8])
def test_stalled_then_solvable(ctx, solver, precision, cut):
    import babelsim_b200 as bsg
    rng = np.random.default_rng(int(10 * cut))
    poly = meshgen.hex_box(26, 26, 26, flat=True)
    own, nbr = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64)
    inner, n = nbr >= 0, poly.n_cells

    def matrix(c):
        d = np.full(n, 1e-2)
        np.add.at(d, own[inner], c[inner])
        np.add.at(d, nbr[inner], c[inner])
        return d, -c
    c = np.where(inner, np.exp(0.3 * rng.standard_normal(len(own))), 0.0)
    cut_d, cut_up = matrix(np.where(rng.random(len(own)) < cut, 0.0, c))
    d, up = matrix(c)
    b = rng.standard_normal(n)
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    system = bsg.LinearSystem(mesh)
    cfg = bsg.solver_config(solver, "hypre", 1e-30, RTOL, 2000, precision=precision)
    for _ in range(2):  # the second call brings the same matrix: nothing changed, and still no hierarchy
        with pytest.raises(bsg.BsgError, match="coarsening stalled"):
            system.solve(cfg, cut_d, cut_up, cut_up, b)
    for _ in range(2):
        x, res = system.solve(cfg, d, up, up, b)
        y = d * x
        np.add.at(y, own[inner], up[inner] * x[nbr[inner]])
        np.add.at(y, nbr[inner], up[inner] * x[own[inner]])
        assert res[0].status == 0
        assert np.linalg.norm(b - y) <= 1.01 * RTOL * np.linalg.norm(b)
    system.close()
    mesh.close()
