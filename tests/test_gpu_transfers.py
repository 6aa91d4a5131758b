"""Host transfers of states, gradients and single passes come back as they were set, at the sizes
where their paths change: one cell to a few, and both sides of the small-state limit."""
import numpy as np
import pytest

from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import Mesh, build_voronoi, random_generators

pytestmark = pytest.mark.gpu


def _mesh(dim, n):
    if n > 1:
        return build_voronoi(random_generators(n, dim, 3), periodic=False)
    # the unit box as one cell with reflective walls
    x = np.full((1, dim), 0.4)
    wall = [(k, e) for k in range(dim) for e in (0.0, 1.0)]
    mid = np.full((2 * dim, dim), 0.5)
    image = np.repeat(x, 2 * dim, axis=0)
    for f, (k, e) in enumerate(wall):
        mid[f, k] = e
        image[f, k] = 2 * e - x[0, k]
    F = 2 * dim
    return Mesh(dim=dim, periodic=False, cell_pos=x, cell_centroid=np.full((1, dim), 0.5),
                cell_volume=np.ones(1), cell_total_area=np.full(1, float(F)),
                cell_face_offset=np.array([0, F], np.int32),
                cell_face_index=np.arange(F, dtype=np.int32), face_area=np.ones(F),
                face_midpoint=mid, face_left=np.zeros(F, np.int32),
                face_right=np.full(F, -1, np.int32), face_kind=np.full(F, 2, np.int32),
                face_right_pos=image)


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_SPLIT])
@pytest.mark.parametrize("dim,n", [(2, 1), (2, 2), (2, 3), (2, 2_047), (2, 2_049), (2, 5_000),
                                   (3, 1), (3, 12), (3, 1_638), (3, 1_640), (3, 4_001)])
def test_round_trips(cuda_ok, oracle, dim, n, precision):
    from oracle.oracle import Params
    mesh = _mesh(dim, n)
    W = wl.random_field_state(mesh, 4)
    ctx = Context(dim, RiemannSolverFactory.generate("HLLC"), precision)
    fp = FluxPass(ctx, mesh)
    rng = np.random.default_rng(n)
    p = Params(solver="HLLC")
    single = (lambda a: a.astype(np.float32).astype(np.float64)) if precision else (lambda a: a)
    for f in (fp, fp.clone()):
        f.set_primitive(W)
        W1, Q1 = f.state()
        Q = oracle.init_Q(mesh, p, W)
        assert np.array_equal(W1, single(W)) and np.array_equal(Q1, Q)
        V, P = rng.random((n, dim + 2)), rng.random((n, dim + 2))
        f.set_state(V, P)
        W1, Q1 = f.state()
        assert np.array_equal(W1, single(V)) and np.array_equal(Q1, P)
        if precision == L.PREC_FP64:
            g = rng.standard_normal((n, dim, dim + 2))
            f.set_gradients(g)
            assert np.array_equal(f.gradients(), g)
            assert np.array_equal(f.state()[1], P)       # and nothing else
    fp.set_state(W, Q)
    dt = 0.1 * wl.cfl_dt(mesh, W)
    grad, dq, _, rc, _ = fp.flux_pass(dt)
    ograd, odq, _, orc, _ = oracle.flux_pass(mesh, p, dt, W, Q)
    assert rc == orc == 0
    if precision == L.PREC_FP64:
        assert np.array_equal(grad, ograd) and np.array_equal(dq, odq)
    else:
        inner = mesh.face_kind != 2                     # walls: no mass through them, by design
        scale = np.abs(odq).max() + 1e-300
        assert (np.abs(dq - odq)[inner] <= 1e-5 * scale).all()
    fp.close()
    ctx.close()
