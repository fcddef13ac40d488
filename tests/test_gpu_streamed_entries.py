"""Solves on either side of the size at which matrix entries pass L1 by (64 MiB of entries: 72 bytes a row on
a hex mesh in FP64, so the line lies at 932k cells; 48 bytes in FP32, 1.4M cells).

The contract is the accepted true residual, ||b - A x|| <= rtol max(||r0||, ||b||), recomputed in numpy; the
recomputation's own rounding is far below 1e-2 of it, so the tolerance is 1.01 rtol."""
import numpy as np
import pytest

from babelsim_b200 import meshgen

pytestmark = pytest.mark.gpu
RTOL = 1e-8


@pytest.mark.parametrize("shape", [(97, 97, 97), (101, 100, 99), (113, 112, 111)], ids=lambda s: "x".join(map(str, s)))
def test_residual_contract(shape):
    import babelsim_b200 as bsg
    ctx = bsg.Context(0)
    rng = np.random.default_rng(shape)
    poly = meshgen.hex_box(*shape, flat=True)
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    own, nbr = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64)
    inner, n = nbr >= 0, poly.n_cells
    c, flux = np.exp(0.3 * rng.standard_normal(len(own))), rng.standard_normal(len(own))
    for skew in (0.0, 1.0):
        up = np.where(inner, -c + skew * np.minimum(flux, 0.0), 0.0)
        lo = np.where(inner, -c - skew * np.maximum(flux, 0.0), 0.0)
        d = np.full(n, 0.05)
        np.add.at(d, own[inner], -up[inner])
        np.add.at(d, nbr[inner], -lo[inner])
        solves = ([(1, "cg", "hypre", 0), (1, "cg", "hypre", 1)] if skew == 0.0
                  else [(3, "bcgs", "bjacobi", 0), (1, "bcgs", "bjacobi", 0), (3, "bcgs", "bjacobi", 1)])
        for components, ksp, pc, precision in solves:
            b = rng.standard_normal((n, components))
            flat = b if components == 3 else b[:, 0]
            system = bsg.LinearSystem(mesh, components)
            cfg = bsg.solver_config(ksp, pc, 1e-30, RTOL, 3000, precision=precision)
            x, res = system.solve(cfg, d, up, lo, flat, np.zeros_like(flat))
            assert all(r.status == 0 for r in res)
            x = x.reshape(n, components)
            y = d[:, None] * x
            np.add.at(y, own[inner], up[inner, None] * x[nbr[inner]])
            np.add.at(y, nbr[inner], lo[inner, None] * x[own[inner]])
            assert np.all(np.linalg.norm(b - y, axis=0) <= 1.01 * RTOL * np.linalg.norm(b, axis=0))
            system.close()
    mesh.close()
    ctx.close()
