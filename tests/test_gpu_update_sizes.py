"""3D split updates of small launches (eight faces in flight per lane) and of larger ones (three)
add a cell's faces in the same order: a mesh alone, in a small launch, and in a group that fills
more than a block per SM has the same bits."""
import numpy as np
import pytest

from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, Group, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 2_500])
def test_alone_and_in_a_large_group(cuda_ok, n):
    mesh = build_voronoi(random_generators(n, 3, 21), periodic=True)
    assert np.diff(mesh.cell_face_offset).max() > 16       # more than two rounds of eight
    W = wl.random_field_state(mesh, 9)
    dt = 0.1 * wl.cfl_dt(mesh, W)
    ctx = Context(3, RiemannSolverFactory.generate("HLLC"), L.PREC_SPLIT)
    alone = FluxPass(ctx, mesh)
    alone.set_primitive(W)
    alone.step(dt, 3)
    want = alone.state()
    many = [alone.clone() for _ in range(148 * 256 // n + 8)]
    for f in many:
        f.set_primitive(W)
    group = Group(ctx, many, [dt] * len(many))
    group.step(3, graph=False)
    for f in (many[0], many[-1]):
        for a, b in zip(f.state(), want):
            assert np.array_equal(a, b)
    group.close()
    for f in (*many, alone):
        f.close()
    ctx.close()
