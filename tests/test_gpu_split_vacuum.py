"""The split HLLC kernel's vacuum cases at gamma 5/3 (integer powers) and others (a power):
vacuum between the sides, a side that is vacuum already, fans on either side, against the plain-FP64
pass face by face."""
import numpy as np
import pytest

from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [5 / 3, 1.4, 1.1])
@pytest.mark.parametrize("dim", [2, 3])
def test_vacuum_faces(cuda_ok, dim, gamma):
    n = 3_000
    mesh = build_voronoi(random_generators(n, dim, 6), periodic=True)
    rng = np.random.default_rng(7)
    W = np.zeros((n, dim + 2))
    W[:, 0] = np.exp(rng.uniform(-1, 1, n))
    W[:, dim + 1] = 0.01 * np.exp(rng.uniform(-1, 1, n))
    c = np.sqrt(gamma * 0.01)
    # opening at up to about three times the speed at which vacuum appears
    W[:, 1:dim + 1] = rng.standard_normal((n, dim)) * 3 * c / (gamma - 1)
    W[rng.random(n) < 0.05] = 0.0                # cells that are vacuum already
    dt = 0.05 * wl.cfl_dt(mesh, np.maximum(W, 1e-3))
    dq, branch = [], None
    for precision in (0, 1):
        ctx = Context(dim, RiemannSolverFactory.generate("HLLC", gamma=gamma), precision)
        fp = FluxPass(ctx, mesh)
        fp.set_primitive(W)
        _, d, br, rc, _ = fp.flux_pass(dt)
        assert rc == 0
        dq.append(d / (dt * np.where(mesh.face_area > 0, mesh.face_area, 1))[:, None])
        branch = br if precision == 0 else branch
        fp.close()
        ctx.close()
    on = mesh.face_area > 0
    top = np.abs(dq[0][on]).max(0)
    top[1:dim + 1] = top[1:dim + 1].max()
    power = 2 / (gamma - 1)
    for kind in (2, 3, 4):                       # right vacuum, left vacuum, vacuum between
        sel = on & ((branch & 7) == kind)
        assert sel.sum() > 20
        # half an ulp in each of the fan base's few operations, times its power, on top of the
        # predicted states' own round-off (1e-6 of the largest flux)
        err = np.abs(dq[1][sel] - dq[0][sel]) / top
        assert err.max() <= 1e-6 + 4 * power * 2.0**-24
