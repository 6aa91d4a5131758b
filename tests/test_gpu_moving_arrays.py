"""Moving and local steps give the same bits whether the moving arrays are set aside in the mesh's
block (small meshes) or allocated on first use, and in either order of the two kinds of step."""
import numpy as np
import pytest

from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_SPLIT])
@pytest.mark.parametrize("dim,n", [(2, 400), (2, 13_400), (3, 300), (3, 4_500)])
def test_moving_and_local_steps_in_either_order(cuda_ok, dim, n, precision):
    mesh = build_voronoi(random_generators(n, dim, 13), periodic=True)
    small = 8 * dim * (2 * n + mesh.n_faces) <= 1 << 20
    assert small == (n < 1_000)
    x = 2 * np.pi * mesh.cell_pos
    W = np.ones((n, dim + 2))
    W[:, 0] += 0.3 * np.sin(x[:, 0])
    W[:, 1:dim + 1] = 0.2 * np.sin(np.roll(x, 1, axis=1))
    dt = 0.05 * wl.cfl_dt(mesh, W)
    ctx = Context(dim, RiemannSolverFactory.generate("Exact"), precision)
    zero = np.zeros(n, np.uint64)

    def local(fp):
        fp.set_primitive(W)
        fp.set_timesteps(zero, zero)
        fp.run_local(640 * dt, 2)
        return fp.state()

    def moving(fp):
        fp.set_primitive(W)
        return fp.step_moving(dt, True), *fp.state()

    a, b = FluxPass(ctx, mesh), FluxPass(ctx, mesh)
    la = local(a)                  # before any face velocity
    ma = moving(a)
    mb = moving(b)
    for p, q in zip(ma, mb):
        assert np.array_equal(p, q)
    for p, q in zip(local(a), local(b)):      # both with the velocities of the moving step
        assert np.array_equal(p, q)
    c = FluxPass(ctx, mesh)
    for p, q in zip(la, local(c)):
        assert np.array_equal(p, q)
    for f in (a, b, c):
        f.close()
    ctx.close()
