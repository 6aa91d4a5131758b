"""The error record names the lowest failing face, as the reference's ascending face loop would,
also when a launch of its own solves that face after others have failed."""
import numpy as np
import pytest

from oracle.oracle import Params
from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    m = build_voronoi(random_generators(25_600, 2, 17), periodic=True)
    assert m.n_faces > 2 * 148 * 256        # the listed faces are a launch of their own
    return m


def _failure(mesh, W, solver, precision, dt, **kw):
    ctx = Context(2, RiemannSolverFactory.generate(solver, **kw), precision)
    fp = FluxPass(ctx, mesh)
    fp.set_primitive(W)
    with pytest.raises(L.SfxError) as e:
        fp.step(dt, 2)
    fp.close()
    ctx.close()
    return e.value.status, e.value.index


def test_listed_face_below_a_failed_one(cuda_ok, oracle, mesh):
    """a tolerance no iteration can meet fails the faces around the first cells, which are listed
    (f(0) above the cutoff); a NaN cell at the mesh's end fails in the first launch"""
    n = mesh.n_cells
    rng = np.random.default_rng(1)
    W = np.zeros((n, 4))
    W[:, 0], W[:, 3] = 1.0, 0.1
    W[:200, 1] = 0.5 * rng.uniform(-1, 1, 200)
    W[:200, 3] = 0.1 * np.exp(0.5 * rng.uniform(-1, 1, 200))
    dt = 0.1 * wl.cfl_dt(mesh, W)
    W[-5, 3] = np.nan
    p = Params(solver="Exact", tolerance=1e-17)
    *_, rc, bad = oracle.flux_pass(mesh, p, dt, W, oracle.init_Q(mesh, p, W))
    assert (rc, bad) == (L.SFX_ERR_NOCONV, 0)
    assert _failure(mesh, W, "Exact", 0, dt, tolerance=1e-17) == (rc, bad)


@pytest.mark.parametrize("solver", ["Exact", "HLLC"])
@pytest.mark.parametrize("precision", [0, 1])
def test_many_failing_faces(cuda_ok, oracle, mesh, solver, precision):
    W = wl.random_field_state(mesh, 23)
    dt = 0.1 * wl.cfl_dt(mesh, W)
    W[np.abs(mesh.cell_pos - 0.5).max(1) < 0.45, 0] = np.nan
    p = Params(solver=solver)
    *_, rc, bad = oracle.flux_pass(mesh, p, dt, W, oracle.init_Q(mesh, p, W))
    assert rc != 0 and bad > 0
    for _ in range(5):
        assert _failure(mesh, W, solver, precision, dt)[1] == bad
