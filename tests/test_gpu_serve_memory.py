"""The server's admission estimate bounds what a resident solve holds on the device, alone and as a member of a
batch, in every pressure precision.  No tolerance: it is a bound."""
import numpy as np
import pytest

from babelsim_b200 import meshgen, serve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import babelsim_b200 as bsg
    c = bsg.Context(0)
    _held(c, [meshgen.hex_box(8, 8, 8, flat=True)], 0)   # kernels are loaded on first use
    _held(c, [meshgen.hex_box(8, 8, 8, flat=True)] * 2, 0)
    yield c
    c.close()


def _held(ctx, meshes, precision):
    import babelsim_b200 as bsg
    import torch
    before = torch.cuda.mem_get_info()[0]
    poly, cells, patches = meshgen.concatenate(meshes) if len(meshes) > 1 else (meshes[0], None, [0])
    mesh = bsg.Mesh.from_polyhedral(ctx, poly)
    opts = bsg.options("linear", "greenGauss", "upwind", "orthogonal")
    sim = bsg.Simple(mesh, 1.0, 1e-2, 0.7, 0.3, 1, 1e-6, 1e-5, 1e-5, 1e-5, opts, opts,
                     bsg.solver_config("bcgs", "bjacobi", 1e-14, 1e-8, 1000),
                     bsg.solver_config("cg", "hypre", 1e-14, 1e-8, 1000, precision=precision))
    if len(meshes) > 1:
        sim.set_segments(cells, [1e-2] * len(meshes))
    for k in range(len(meshes)):
        for p in range(6):
            sim.set_boundary("U", patches[k] + p, "fixedValue", (1.0 if p == 3 else 0.0, 0.0, 0.0))
            sim.set_boundary("p", patches[k] + p, "zeroGradient")
    sim.set_fields(np.zeros((mesh.n_cells, 3)), np.zeros(mesh.n_cells))
    sim.iterate(2)
    held = before - torch.cuda.mem_get_info()[0]
    sim.close()
    mesh.close()
    return held


@pytest.mark.parametrize("members", [1, 4])
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("shape", [8, 24, 48, "voronoi"])
def test_estimate_bounds_a_resident_solve(ctx, shape, precision, members):
    if precision == 1 and members > 1:
        pytest.skip("batches take precision 0 and 2")
    mesh = meshgen.voronoi_cube(20, 0.3, 1) if shape == "voronoi" else meshgen.hex_box(shape, shape, shape, flat=True)
    estimate = members * serve.device_bytes(mesh.n_cells, len(mesh.owner))
    assert _held(ctx, [mesh] * members, precision) <= estimate
