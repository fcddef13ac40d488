"""BiCGStab through the linear-system seam at the sizes where its placement changes (a cluster, the grid
with rows and vectors on chip, the grid streaming), for one and three right-hand sides, from a
zero and from a given guess, in FP64 and with FP32 inner iterations.

The contract is the accepted true residual per component, ||b - A x|| <= rtol max(||r0||, ||b||), recomputed
in numpy; the recomputation's own rounding is far below 1e-2 of it, so the tolerance is 1.01 rtol."""
import numpy as np
import pytest

from babelsim_b200 import meshgen

pytestmark = pytest.mark.gpu
RTOL = 1e-10
SHAPES = [(1, 1, 1), (5, 3, 2), (16, 16, 16), (21, 20, 20), (47, 46, 45), (200, 150, 1), (72, 71, 70)]


@pytest.fixture(scope="module")
def ctx():
    import babelsim_b200 as bsg
    c = bsg.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("components,precision,warm", [(3, 0, False), (1, 0, False), (3, 0, True), (1, 0, True),
                                                       (3, 1, False), (1, 1, False)])
def test_residual_contract(ctx, shape, components, precision, warm):
    import babelsim_b200 as bsg
    rng = np.random.default_rng([*shape, components, precision])
    poly = meshgen.hex_box(*shape, flat=True)
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    own, nbr = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64)
    inner, n = nbr >= 0, poly.n_cells
    c, flux = np.exp(0.3 * rng.standard_normal(len(own))), rng.standard_normal(len(own))
    up = np.where(inner, -c + np.minimum(flux, 0.0), 0.0)
    lo = np.where(inner, -c - np.maximum(flux, 0.0), 0.0)
    d = np.full(n, 0.05)
    np.add.at(d, own[inner], -up[inner])
    np.add.at(d, nbr[inner], -lo[inner])

    def residual(x, b):
        y = d[:, None] * x
        np.add.at(y, own[inner], up[inner, None] * x[nbr[inner]])
        np.add.at(y, nbr[inner], lo[inner, None] * x[own[inner]])
        return np.linalg.norm(b - y, axis=0)
    b = rng.standard_normal((n, components))
    x0 = rng.standard_normal((n, components)) if warm else np.zeros((n, components))
    flat = (lambda a: a) if components == 3 else (lambda a: a[:, 0])
    system = bsg.LinearSystem(mesh, components)
    cfg = bsg.solver_config("bcgs", "bjacobi", 1e-30, RTOL, 3000, warm_start=warm, precision=precision)
    x, res = system.solve(cfg, d, up, lo, flat(b), flat(x0))
    assert all(r.status == 0 for r in res)
    bound = 1.01 * RTOL * np.maximum(np.linalg.norm(b, axis=0), residual(x0, b))
    assert np.all(residual(x.reshape(n, components), b) <= bound)
    again, _ = system.solve(cfg, d, up, lo, flat(b), flat(x0))
    assert np.array_equal(x, again)  # fixed-order reductions: the same bits
    system.close()
    mesh.close()
