"""FP32 inner BiCGStab inside FP64 refinement (precision 1) against a numpy restatement of its arithmetic.

The refinement accepts the first iterate under its target, so what the FP32 iterations round decides which
iterate that is, and two kernels that round differently return solutions that differ by a part of the target:
fields of one mixed outer iteration then no longer agree with the ones it gave before.  The restatement
rounds every FP32 operation as the solver is meant to (row sums in entry order by fused multiply-adds with
the diagonal last, rho = r0 . r of the residual that is kept, sums in FP64).  Two expressions may be
contracted either way (the diagonal's product, the pair of products in the solution update); one of the four
ways has to match.

Tolerance 5e-11 relative, on 12x11x10 to 33x32x31 cells at rtol 1e-10: the order of FP64 sums moves the
restated solution by up to 1e-11 (an FP32 rounding of the residual falls the other way), rounding that is
not the solver's (rho from the unrounded residual, the diagonal first) by 1.1e-10 or more."""
import itertools

import numpy as np
import pytest

from babelsim_b200 import meshgen

pytestmark = pytest.mark.gpu
RTOL = 1e-10
F = np.float32


@pytest.fixture(scope="module")
def ctx():
    import babelsim_b200 as bsg
    c = bsg.Context(0)
    yield c
    c.close()


def _fma(a, b, c):
    # the product of two FP32 values is exact in FP64
    return (a.astype(float) * np.asarray(b, float) + np.asarray(c, float)).astype(F)


def _rows(poly, up, lo):
    """Padded rows: entries of a cell in the order of its faces, interior faces sorted by owner."""
    own, nbr, n = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64), poly.n_cells
    f = np.nonzero(nbr >= 0)[0]
    f = f[np.argsort(own[f], kind="stable")]
    row, col = np.stack([own[f], nbr[f]], 1).ravel(), np.stack([nbr[f], own[f]], 1).ravel()
    val = np.stack([up[f], lo[f]], 1).ravel()
    o = np.argsort(row, kind="stable")
    row, col, val = row[o], col[o], val[o]
    k = np.arange(len(row)) - np.searchsorted(row, row)
    cols, vals = np.tile(np.arange(n)[:, None], (1, k.max() + 1)), np.zeros((n, k.max() + 1))
    cols[row, k], vals[row, k] = col, val
    return cols, vals


def _refined(cols, vals, d, b, fused_diagonal, first_product):
    """b's solution as precision 1 computes it (one right-hand side)."""
    v32, d32 = vals.astype(F), d.astype(F)
    rd = F(1) / d32

    def product(y):
        a = np.zeros(len(d), F)
        for k in range(cols.shape[1]):
            a = _fma(v32[:, k], y[cols[:, k]], a)
        return _fma(d32, y, a) if fused_diagonal else d32 * y + a

    def dot(u, w):
        return float(u.astype(float) @ w.astype(float))
    x = np.zeros(len(d))
    res, target = b.copy(), RTOL * np.linalg.norm(b)
    for _ in range(12):
        norm = np.linalg.norm(res)
        if norm <= target:
            break
        stop = (max(1e-5, 0.5 * target / norm) * norm) ** 2
        r = r0 = res.astype(F)
        dx = p = v = np.zeros(len(d), F)
        rho, beta, omega = dot(r, r), 0.0, 1.0
        while True:
            p = _fma(_fma(v, F(-omega), p), F(beta), r)
            ph = p * rd
            v = product(ph)
            alpha = rho / dot(r0, v)
            r = _fma(v, F(-alpha), r)
            sh = r * rd
            if dot(r, r) <= stop:
                dx = _fma(ph, F(alpha), dx)
                break
            t = product(sh)
            omega = dot(t, r) / dot(t, t)
            dx = dx + (_fma(ph, F(alpha), F(omega) * sh) if first_product else _fma(sh, F(omega), F(alpha) * ph))
            r = _fma(t, F(-omega), r)
            if dot(r, r) <= stop:
                break
            new = dot(r0, r)
            beta, rho = (new / rho) * (alpha / omega), new
        x = x + dx.astype(float)
        res = b - (d * x + (vals * x[cols]).sum(1))
    return x


@pytest.mark.parametrize("components", [1, 3])
@pytest.mark.parametrize("shape", [(12, 11, 10), (16, 16, 16), (33, 32, 31)], ids=lambda s: "x".join(map(str, s)))
def test_inner_solver_rounds_as_stated(ctx, shape, components):
    import babelsim_b200 as bsg
    rng = np.random.default_rng([*shape, 0])
    poly = meshgen.hex_box(*shape, flat=True)
    own, nbr = np.asarray(poly.owner, np.int64), np.asarray(poly.neighbour, np.int64)
    inner, n = nbr >= 0, poly.n_cells
    c, flux = np.exp(0.3 * rng.standard_normal(len(own))), rng.standard_normal(len(own))
    up = np.where(inner, -c + np.minimum(flux, 0.0), 0.0)
    lo = np.where(inner, -c - np.maximum(flux, 0.0), 0.0)
    d = np.full(n, 0.5)
    np.add.at(d, own[inner], -up[inner])
    np.add.at(d, nbr[inner], -lo[inner])
    b = rng.standard_normal((n, components))
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    system = bsg.LinearSystem(mesh, components)
    cfg = bsg.solver_config("bcgs", "bjacobi", 1e-30, RTOL, 3000, precision=1)
    x, res = system.solve(cfg, d, up, lo, b if components == 3 else b[:, 0])
    system.close()
    mesh.close()
    assert all(r.status == 0 for r in res)
    x = x.reshape(n, components)
    cols, vals = _rows(poly, up, lo)
    for k in range(components):  # each component is its own code, contracted in its own way
        off = [np.linalg.norm(x[:, k] - s) / np.linalg.norm(s)
               for s in (_refined(cols, vals, d, b[:, k].copy(), *ways)
                         for ways in itertools.product((True, False), repeat=2))]
        assert min(off) <= 5e-11, off
