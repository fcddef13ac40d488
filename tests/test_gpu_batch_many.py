"""Batches of more members than one launch used to hold: 33 to 150 small cases of six kinds side by side.

Each member gives what its case gives alone to 1e-9 relative L2 after two outer iterations (only the order of
dot-product sums differs, as in test_gpu_batch.py), and members that leave SMs idle share one launch per
solve: 128 at most, which is what one kernel argument holds."""
import numpy as np
import pytest

from babelsim_b200 import meshgen
from helpers import rel_l2

pytestmark = pytest.mark.gpu
KINDS = [((2, 2, 2), 1.0, 1e-2), ((5, 4, 3), 1.0, 2e-2), ((6, 6, 6), 2.0, 1e-2), ((9, 7, 5), 0.5, 1e-2),
         ((8, 8, 8), 1.0, 5e-3), ((11, 10, 9), 1.0, 1e-2)]


@pytest.fixture(scope="module")
def ctx():
    import babelsim_b200 as bsg
    c = bsg.Context(0)
    yield c
    c.close()


def _run(ctx, kinds, precision):
    import babelsim_b200 as bsg
    poly, cells, patches = meshgen.concatenate([meshgen.hex_box(*KINDS[k][0], flat=True) for k in kinds])
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    opts = bsg.options("linear", "greenGauss", "upwind", "orthogonal")
    sim = bsg.Simple(mesh, 1.0, 1e-2, 0.7, 0.3, 1, 1e-12, 1e-12, 1e-12, 1e-12, opts, opts,
                     bsg.solver_config("bcgs", "bjacobi", 1e-15, 1e-10, 2000),
                     bsg.solver_config("cg", "hypre", 1e-15, 1e-10, 5000, precision=precision))
    sim.set_segments(cells, [KINDS[k][2] for k in kinds])
    for i, k in enumerate(kinds):
        for p in range(6):
            sim.set_boundary("U", patches[i] + p, "fixedValue", (KINDS[k][1] if p == 3 else 0.0, 0.0, 0.0))
            sim.set_boundary("p", patches[i] + p, "zeroGradient")
    sim.set_fields(np.zeros((mesh.n_cells, 3)), np.zeros(mesh.n_cells))
    ctx.profile(True)
    sim.iterate(2)
    report = ctx.profile_report()
    ctx.profile(False)
    U, p, _ = sim.fields()
    sim.close()
    mesh.close()
    return U, p, cells, report


@pytest.mark.parametrize("members,precision", [(33, 0), (150, 0), (129, 2)])
def test_many_members_match_their_solo_runs(ctx, members, precision):
    kinds = [k % len(KINDS) for k in range(members)]
    U, p, cells, report = _run(ctx, kinds, precision)
    few = _run(ctx, [0], precision)[3]
    launches = 1 if members <= 128 else 2
    assert report["pcg_amg_persistent_batch"][0] <= launches * few["pcg_amg_persistent_batch"][0] + 2  # + 2 restarts
    for k in range(len(KINDS)):
        U1, p1, _, _ = _run(ctx, [k], precision)
        for i in range(k, members, len(KINDS)):
            assert rel_l2(U[cells[i]:cells[i + 1]], U1) < 1e-9
            assert rel_l2(p[cells[i]:cells[i + 1]], p1) < 1e-9
