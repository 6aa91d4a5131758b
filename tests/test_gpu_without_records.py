"""A plain-FP64 mesh whose records do not fit in the device's free memory is stored without them
and gives the same bits: steps, moving and local steps, single passes, clones, packed cells."""
import numpy as np
import pytest

from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


def _results(fp, mesh, W, dt, clones):
    import torch
    out = []
    for f in [fp, *clones]:
        f.set_primitive(W)
        grad, dq, branch, rc, _ = f.flux_pass(dt)
        assert rc == 0
        st = f.step(dt, 2)
        out += [grad, dq, branch, *f.state(), np.array(st.totals[:f.S])]
        f.set_gradients(grad)
        assert np.array_equal(f.gradients(), grad)
        f.set_state(*f.state())
        f.step(dt, 1)
        idx = torch.arange(0, mesh.n_cells, 7, dtype=torch.int32, device="cuda")
        buf = torch.zeros(idx.numel(), f.S + 1, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        f.pack_cells(idx, buf)
        f.ctx.synchronize()
        changed = buf * 1.01
        torch.cuda.synchronize()
        f.unpack_cells(idx, changed)
        f.ctx.synchronize()
        f.step(dt, 1)
        out += [buf.cpu().numpy(), *f.state()]
        zero = np.zeros(mesh.n_cells, np.uint64)
        f.set_primitive(W)
        f.set_timesteps(zero, zero)
        tick = f.run_local(64 * dt, 3)
        out += [*f.state(), f.gradients(), np.array(tick)]
    if fp.ctx.solver.tag() == "EXAC":   # HLLC's moving step of this mesh goes negative, as the reference's
        fp.set_primitive(W)
        out += [fp.step_moving(dt, mesh.periodic), *fp.state()]
    return out


@pytest.mark.parametrize("dim,n,solver,periodic", [(3, 30_000, "Exact", True),
                                                   (2, 120_000, "Exact", False),
                                                   (2, 120_000, "HLLC", True)])
def test_without_records(cuda_ok, dim, n, solver, periodic):
    import torch
    mesh = build_voronoi(random_generators(n, dim, 29), periodic=periodic)
    # subsonic waves: the moving step follows them
    x = 2 * np.pi * mesh.cell_pos
    W = np.ones((n, dim + 2))
    W[:, 0] += 0.3 * np.sin(x[:, 0])
    W[:, 1:dim + 1] = 0.2 * np.sin(np.roll(x, 1, axis=1))
    W[:, dim + 1] += 0.2 * np.cos(x[:, dim - 1])
    dt = 0.1 * wl.cfl_dt(mesh, W)
    ctx = Context(dim, RiemannSolverFactory.generate(solver), L.PREC_FP64)
    fp = FluxPass(ctx, mesh)
    clone = fp.clone()
    need = L.lib().sfx_mesh_device_bytes(dim, mesh.n_cells, mesh.n_faces, mesh.nnz, L.PREC_FP64)
    want = _results(fp, mesh, W, dt, [clone])
    clone.close()
    fp.close()
    torch.cuda.empty_cache()

    def leave(size):
        """hold the device's free memory but for `size` bytes"""
        return torch.empty(torch.cuda.mem_get_info()[0] - size, dtype=torch.uint8, device="cuda")

    held = leave(int(0.8 * need))
    fp = FluxPass(ctx, mesh)
    used = int(0.8 * need) - torch.cuda.mem_get_info()[0]
    assert used < 0.6 * need                  # without its records
    del held
    torch.cuda.empty_cache()
    size = int(0.92 * fp.clone_bytes(L.PREC_FP64))
    held = leave(size)
    clone = fp.clone()                         # as its base
    del held
    torch.cuda.empty_cache()
    got = _results(fp, mesh, W, dt, [clone])
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    clone.close()
    fp.close()
    # a clone without records of a mesh with them
    fp = FluxPass(ctx, mesh)
    held = leave(size)
    clone = fp.clone()
    del held
    torch.cuda.empty_cache()
    for a, b in zip(_results(fp, mesh, W, dt, [clone]), want):
        assert np.array_equal(a, b)
    clone.close()
    fp.close()
    ctx.close()
