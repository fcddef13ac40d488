"""CG + AMG from a given guess in FP64 at every placement of the solver, complete and with cut couplings, and
without one where couplings are cut: every case has to solve.  Only a system whose couplings leave more than 2048
parts has to be refused, which the test counts for itself.  (Pairwise matching also gives up, after twelve levels,
on large systems with many cut couplings that leave fewer parts; the 358k-cell box has a tenth cut at most.)

Contract and tolerance as in test_gpu_tree.py: the accepted true residual recomputed in numpy, 1.01 rtol."""
import numpy as np
import pytest

from babelsim_b200 import meshgen
from test_gpu_tree import RTOL, SHAPES, _matrix, _residual

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import babelsim_b200 as bsg
    c = bsg.Context(0)
    yield c
    c.close()


def _parts(n, up, inner, own, nbr):
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    k = inner & (up != 0.0)
    return connected_components(coo_matrix((np.ones(int(k.sum())), (own[k], nbr[k])), shape=(n, n)))[0]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("cut,precision,warm", [(0.0, 0, True), (0.2, 0, True), (0.3, 0, True), (0.3, 0, False),
                                                (0.2, 1, True), (0.05, 2, False), (0.9, 0, True)])
def test_solves_or_is_refused_for_its_parts(ctx, shape, cut, precision, warm):
    import babelsim_b200 as bsg
    if cut < 0.5 and np.prod(shape) > 100000:
        cut = min(cut, 0.1)
    rng = np.random.default_rng([*shape, int(10 * cut), precision, 1])
    poly = meshgen.hex_box(*shape, flat=True)
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    d, up, *pattern = _matrix(poly, cut, rng)
    b = rng.standard_normal(poly.n_cells)
    x0 = rng.standard_normal(poly.n_cells) if warm else None
    system = bsg.LinearSystem(mesh)
    cfg = bsg.solver_config("cg", "hypre", 1e-30, RTOL, 5000, warm_start=warm, precision=precision)
    if _parts(poly.n_cells, up, *pattern) > 2048:
        assert cut > 0.5  # the cases above it are meant to be solved
        with pytest.raises(bsg.BsgError, match="coarsening stalled"):
            system.solve(cfg, d, up, up, b, x0)
    else:
        for _ in range(2):  # the second matrix meets the first one's (lagged) coarse levels
            x, res = system.solve(cfg, d, up, up, b, x0)
            scale = np.linalg.norm(b) if not warm else max(np.linalg.norm(b), _residual(x0, b, d, up, *pattern))
            assert res[0].status == 0
            assert _residual(x, b, d, up, *pattern) <= 1.01 * RTOL * scale
            d = d * (1.0 + 0.1 * rng.random(poly.n_cells))
    system.close()
    mesh.close()
