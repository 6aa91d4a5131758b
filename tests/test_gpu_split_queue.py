"""The split pass's queue of faces starts empty in every step, also of a part with faces and no
cells of its own (no gradient launch)."""
import numpy as np
import pytest

from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_queue_is_emptied_without_a_gradient_launch(cuda_ok, dim):
    n = 600
    mesh = build_voronoi(random_generators(n, dim, 5), periodic=False)
    # densities below the range of the FP32 iteration: those faces are queued in every step
    W = np.zeros((n, dim + 2))
    W[:, 0] = np.where(mesh.cell_pos[:, 0] < 0.5, 1.0, 1e-13)
    W[:, dim + 1] = 0.1 * W[:, 0]
    ctx = Context(dim, RiemannSolverFactory.generate("Exact"), 1)
    fp = FluxPass(ctx, mesh)
    fp.set_primitive(W)
    dt = 1e-4 * wl.cfl_dt(mesh, W)
    fp.step(dt, 1)
    before = fp.state()
    fp.set_ranges(0, mesh.n_faces, 0)
    # more queued faces over the steps than the queue has room for
    st = fp.step(dt, 8)
    assert st.status == 0
    after = fp.state()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
    fp.close()
    ctx.close()
