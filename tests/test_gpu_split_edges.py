"""Branches of the split pass's kernels that the workloads reach rarely: vacuum faces of the
HLLC kernel (solved in FP64 by the queue), cells whose face count leaves remainders in the
gradient and update loops, meshes smaller than a block."""
import numpy as np
import pytest

from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


def _run(mesh, W0, solver, precision, dt, steps, lanes=None):
    ctx = Context(mesh.dim, RiemannSolverFactory.generate(solver), precision)
    fp = FluxPass(ctx, mesh)
    if lanes:
        fp.set_lanes(lanes)
    fp.set_primitive(W0)
    fp.step(dt, steps)
    out = fp.state()
    fp.close()
    ctx.close()
    return out


def _close(a, b, scale):
    """1e-6 relative L1 per field, the split pass's stated error; momentum against the
    momentum a sound wave carries (it starts at rest or cancels)"""
    err = np.abs(a - b).sum(0)
    ref = np.maximum(np.abs(b).sum(0), scale)
    assert np.all(err <= 1e-6 * ref), err / ref


@pytest.mark.parametrize("dim", [2, 3])
def test_hllc_vacuum_faces(dim):
    """two gases flying apart faster than they can expand: vacuum opens at the faces between
    them, and its fan is sampled.  Per face, walls left out: the split pass lets no mass
    through a wall, where the reference's HLLC does when a supersonic flow meets one"""
    n = 600
    mesh = build_voronoi(random_generators(n, dim, 5), periodic=False)
    W = np.zeros((n, dim + 2))
    left = mesh.cell_pos[:, 0] < 0.5
    W[:, 0] = np.where(left, 1.0, 0.5)
    W[:, dim + 1] = 0.1
    W[:, 1] = np.where(left, -3.0, 3.0)
    dt = 0.2 * wl.cfl_dt(mesh, W)
    dq, branch = [], None
    for precision in (0, 1):
        ctx = Context(dim, RiemannSolverFactory.generate("HLLC"), precision)
        fp = FluxPass(ctx, mesh)
        fp.set_primitive(W)
        _, d, br, rc, _ = fp.flux_pass(dt)
        assert rc == 0
        dq.append(d)
        branch = br if precision == 0 else branch
        fp.close()
        ctx.close()
    inner = mesh.face_kind != 2
    vacuum = inner & ((branch & 7) == 4)
    assert vacuum.sum() > 10
    # the fan's density is a power of a difference of order one: its round-off, times the
    # power 5, against the largest flux
    tol = 5 * 2.0**-22
    top = np.abs(dq[0][inner]).max(0).max()
    assert np.abs(dq[1][vacuum] - dq[0][vacuum]).max() <= tol * top
    c = np.sqrt(wl.GAMMA * W[:, dim + 1] / W[:, 0])
    _close(dq[1][inner], dq[0][inner], dt * (mesh.face_area[inner]).sum() * c.max())


@pytest.mark.parametrize("dim,n", [(2, 5), (2, 33), (2, 257), (3, 5), (3, 37), (3, 130)])
@pytest.mark.parametrize("solver", ["Exact", "HLLC"])
def test_small_and_ragged_meshes_at_every_lane_count(dim, n, solver):
    mesh = build_voronoi(random_generators(n, dim, 3 + n), periodic=False)
    W = wl.random_field_state(mesh, n)
    W[:, 1:dim + 1] *= 0.3                       # velocities of both signs near zero
    dt = 0.2 * wl.cfl_dt(mesh, W)
    W64, Q64 = _run(mesh, W, solver, 0, dt, 3)
    scale = (W64[:, 0] * mesh.cell_volume * np.sqrt(wl.GAMMA * W64[:, -1] / W64[:, 0])).sum()
    for lanes in (1, 2, 4, 16):
        _close(_run(mesh, W, solver, 1, dt, 3, lanes)[1], Q64, scale)


@pytest.mark.parametrize("n", [50_000, 51_500])
def test_2d_hllc_kernels_on_both_sides_of_one_wave(n):
    """the default face variant, 64 registers below 151,552 faces and 48 above, has the bits of
    the 80-register variant 1"""
    mesh = build_voronoi(random_generators(n, 2, 5), periodic=True)
    assert (mesh.n_faces > 4 * 148 * 256) == (n == 51_500)
    W = wl.random_field_state(mesh, 5)
    ctx = Context(2, RiemannSolverFactory.generate("HLLC"), 1)
    fp = FluxPass(ctx, mesh)
    out = []
    for variant in (0, 1):
        fp.set_face_variant(variant)
        fp.set_primitive(W)
        out.append(fp.flux_pass(0.1 * wl.cfl_dt(mesh, W))[1])
    assert np.array_equal(out[0], out[1])
    fp.close()
    ctx.close()
