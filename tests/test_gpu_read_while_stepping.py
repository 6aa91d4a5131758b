"""Reading a mesh's state, gradients or totals on one stream while its steps are queued on another
leaves the steps as they are."""
import ctypes as C

import numpy as np
import pytest

from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_SPLIT])
@pytest.mark.parametrize("n", [1_000, 20_000])
def test_reads_beside_steps(cuda_ok, precision, n):
    import torch
    mesh = build_voronoi(random_generators(n, 2, 33), periodic=True)
    W = wl.random_field_state(mesh, 2)
    W[:, 1:3] *= 0.3
    dt = 0.05 * wl.cfl_dt(mesh, W)
    ctx = Context(2, RiemannSolverFactory.generate("Exact"), precision)
    fp = FluxPass(ctx, mesh)
    fp.set_primitive(W)
    fp.step(dt, 60)
    want = fp.state()
    fp.set_primitive(W)
    ctx.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    lib = L.lib()
    L.check(lib.sfx_ctx_set_stream(ctx.h, C.c_void_p(a.cuda_stream)), "set_stream")
    fp.step(dt, 60, stats=False)              # queued, not waited for
    L.check(lib.sfx_ctx_set_stream(ctx.h, C.c_void_p(b.cuda_stream)), "set_stream")
    for _ in range(4):
        fp.state()
        fp.totals()
        if precision == L.PREC_FP64:
            fp.gradients()
    a.synchronize()
    for got, ref in zip(fp.state(), want):
        assert np.array_equal(got, ref)
    L.check(lib.sfx_ctx_set_stream(ctx.h, None), "set_stream")
    fp.close()
    ctx.close()
