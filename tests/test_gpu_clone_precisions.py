"""Clones across precisions: a plain-FP64 clone of a split mesh gives the bits of an FP64 upload of
the same mesh, and a split clone of that clone those of the split mesh."""
import numpy as np
import pytest

from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


def _mesh(dim, periodic, shuffled):
    mesh = build_voronoi(random_generators(600, dim, 41), periodic=periodic)
    if shuffled:
        # cells that do not list their faces in ascending order
        rng = np.random.default_rng(2)
        off = mesh.cell_face_offset
        for i in range(mesh.n_cells):
            rng.shuffle(mesh.cell_face_index[off[i]:off[i + 1]])
    return mesh


@pytest.mark.parametrize("solver", ["Exact", "HLLC"])
@pytest.mark.parametrize("dim,periodic,shuffled", [(2, False, False), (2, True, False),
                                                   (3, False, True), (3, True, False),
                                                   (2, True, True)])
def test_clones_across_precisions(cuda_ok, dim, periodic, shuffled, solver):
    mesh = _mesh(dim, periodic, shuffled)
    W = wl.random_field_state(mesh, 5)
    dt = 0.2 * wl.cfl_dt(mesh, W)
    c64, c32 = (Context(dim, RiemannSolverFactory.generate(solver), p)
                for p in (L.PREC_FP64, L.PREC_SPLIT))
    base64, base32 = FluxPass(c64, mesh), FluxPass(c32, mesh)
    clone64 = base32.clone(c64)
    again64 = clone64.clone()
    clone32 = clone64.clone(c32)
    last64 = clone32.clone(c64)
    assert base32.clone_bytes(L.PREC_FP64) > base64.clone_bytes(L.PREC_FP64)

    def steps(fp):
        fp.set_primitive(W)
        st = fp.step(dt, 3)
        return [*fp.state(), np.array(st.totals[:fp.S])]

    want = steps(base64)
    for fp in (clone64, again64, last64):
        for a, b in zip(steps(fp), want):
            assert np.array_equal(a, b)
        for f in (fp, base64):
            f.set_primitive(W)
        for a, b in zip(fp.flux_pass(dt)[:3], base64.flux_pass(dt)[:3]):
            assert np.array_equal(a, b)
    for a, b in zip(steps(clone32), steps(base32)):
        assert np.array_equal(a, b)
    for fp in (last64, clone32, again64, clone64, base32, base64):
        fp.close()
    c64.close()
    c32.close()
