"""e2d_step_noalloc above 12000 cells, whose pass A works in tiles with two
threads per cell (a solver of that size takes a list of the faces), against
the CPU oracle, bit for bit: both sides of the line, partial tiles, the largest
mesh, and the options."""
import ctypes

import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d
from gpueularsolver2d_gb300 import _lib
from test_zz_no_alloc import file_order_layout

pytestmark = pytest.mark.gpu


def compare(lib, oracle, ni, nj, iters, **kw):
    import torch
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    p = e2d.default_params(ma=0.6, alpha_deg=1.5, cfl=1.2, **kw)
    x, y, tri = mesh.nodes()
    c = oracle.Case(x, y, tri, oracle.params_from_e2d(p))
    w = c.state()
    dev = [torch.from_numpy(a).cuda() for a in (*file_order_layout(mesh), w.ravel().copy(), np.zeros(iters))]
    topo, S, R, area, state, res = (ctypes.c_void_p(t.data_ptr()) for t in dev)
    epsm = ctypes.c_double(0.0)
    _lib.check(lib.e2d_step_noalloc(len(w), topo, S, R, area, ctypes.byref(p), iters, state, res, ctypes.byref(epsm),
                                    None))
    c.run(iters)
    assert np.array_equal(dev[4].cpu().numpy().reshape(-1, 4), c.state())


@pytest.mark.parametrize("ni,nj", [(75, 80), (77, 78), (101, 61), (150, 107), (128, 128)])  # 12000 to 32768 cells
def test_sizes(lib, oracle, ni, nj):
    compare(lib, oracle, ni, nj, 3)


@pytest.mark.parametrize("kw", [dict(limiter=1), dict(limiter=2), dict(limiter=3), dict(positivity_fix=1),
                                dict(global_dt=1), dict(first_order_iters=2), dict(irs_sweeps=0)])
def test_options(lib, oracle, kw):
    compare(lib, oracle, 101, 61, 5, **kw)
