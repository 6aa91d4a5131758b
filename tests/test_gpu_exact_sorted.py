"""The plain-FP64 exact solver's sorted face kernel and its list of faces above the cutoff: bit
for bit with the CPU oracle at the edges of its blocks (256 faces) and on both sides of the
face count (75,776) from which the list is a launch of its own."""
import numpy as np
import pytest

from oracle.oracle import Params
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu
LIST_FROM = 2 * 148 * 256


@pytest.mark.parametrize("dim,n,cutoff", [
    (2, 3, -5.0), (2, 85, -5.0), (2, 86, -5.0), (2, 700, 1e3), (2, 700, -1e3),
    (2, 25_000, -5.0), (2, 25_600, -5.0), (3, 60, -5.0), (3, 8_800, -5.0), (3, 10_500, -5.0)])
def test_sorted_faces_equal_the_oracle(oracle, dim, n, cutoff):
    mesh = build_voronoi(random_generators(n, dim, 17), periodic=n > 100)
    if n > 1_000:
        assert (mesh.n_faces > LIST_FROM) == (n in (25_600, 10_500))
    W = wl.random_field_state(mesh, 23)
    dt = 0.1 * wl.cfl_dt(mesh, W)
    # cutoffs of +-1000 send every face to Newton's loop alone, and none
    solver = RiemannSolverFactory.generate("Exact", cutoff=cutoff)
    ctx = Context(dim, solver, 0)
    fp = FluxPass(ctx, mesh)
    fp.set_primitive(W)
    _, dq, br, rc, bad = fp.flux_pass(dt)
    p = Params(solver="Exact", cutoff=cutoff)
    _, odq, obr, orc, obad = oracle.flux_pass(mesh, p, dt, W, oracle.init_Q(mesh, p, W))
    assert (rc, bad) == (orc, obad)
    if rc == 0:
        assert np.array_equal(br, obr)
        assert np.array_equal(dq, odq)
    fp.close()
    ctx.close()


def test_face_list_is_emptied_without_a_gradient_launch():
    """a part with faces and no cells of its own: the list of each step starts empty"""
    mesh = build_voronoi(random_generators(25_600, 2, 17), periodic=True)
    assert mesh.n_faces > LIST_FROM
    W = wl.random_field_state(mesh, 23)
    ctx = Context(2, RiemannSolverFactory.generate("Exact", cutoff=-1e3), 0)   # every face listed
    fp = FluxPass(ctx, mesh)
    fp.set_primitive(W)
    fp.step(0.1 * wl.cfl_dt(mesh, W), 1)
    before = fp.state()
    fp.set_ranges(0, mesh.n_faces, 0)
    st = fp.step(0.1 * wl.cfl_dt(mesh, W), 3)
    assert st.status == 0
    after = fp.state()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
    fp.close()
    ctx.close()
