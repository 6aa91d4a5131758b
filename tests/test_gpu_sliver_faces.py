"""Faces whose area is subnormal in FP32: the split pass takes them as the plain-FP64 pass does,
to the resolution of a subnormal; an area that rounds to zero in FP32 is a zero area to it."""
import dataclasses

import numpy as np
import pytest

from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu
AREAS = [1.3e-38, 1.1e-38, 1e-39, 3e-42, 1.4e-45, 1e-46, 1e-60]


@pytest.mark.parametrize("solver", ["Exact", "HLLC"])
@pytest.mark.parametrize("dim", [2, 3])
def test_subnormal_areas(cuda_ok, dim, solver):
    mesh = build_voronoi(random_generators(400, dim, 9), periodic=False)
    rng = np.random.default_rng(4)
    inner = np.flatnonzero((mesh.face_kind == 0) & (mesh.face_area > 0))
    slivers = rng.choice(inner, 20 * len(AREAS), replace=False)
    mesh.face_area[slivers] = np.tile(AREAS, 20)
    W = wl.random_field_state(mesh, 3)
    W[:, 1:dim + 1] *= 0.3
    dt = 0.2 * wl.cfl_dt(mesh, W)
    dq = []
    rounded = np.where(mesh.face_area.astype(np.float32) == 0, 0.0, mesh.face_area)
    for precision in (0, 1):
        ctx = Context(dim, RiemannSolverFactory.generate(solver), precision)
        fp = FluxPass(ctx, dataclasses.replace(mesh, face_area=rounded) if precision == 0 else mesh)
        fp.set_primitive(W)
        _, d, _, rc, _ = fp.flux_pass(dt)
        assert rc == 0
        dq.append(d)
        fp.set_primitive(W)
        assert fp.step(dt, 2).status == 0
        assert np.isfinite(fp.state()[1]).all()
        fp.close()
        ctx.close()
    a, b = dq[1][slivers], dq[0][slivers]
    flux = np.abs(dq[0][inner] / (dt * mesh.face_area[inner])[:, None]).max()
    # dt A rounded in FP32's subnormal range, its product with the flux rounded again, and the
    # states' relative error of a single face (1e-5, as for the other faces of the split pass)
    scale = dt * mesh.face_area[slivers] * flux
    assert (np.abs(a - b) <= (1e-5 * scale + 2.0**-149 * (1 + flux))[:, None]).all()
