"""FP64 formulas evaluated again with the IEEE operations where an operand is
subnormal (the integer-unit operations take normal numbers and zeros): states
with momenta of 1e-310, and a smoothing coefficient of 1e-310, in finite runs
against the CPU oracle, bit for bit."""
import ctypes

import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d
from gpueularsolver2d_gb300 import _lib
from test_zz_no_alloc import file_order_layout

pytestmark = pytest.mark.gpu

# smoothing in range or not; the reference's limiter and the smooth one
KW = [dict(), dict(irs_eps=1e-310), dict(limiter=1), dict(irs_eps=1e-310, limiter=3, positivity_fix=1)]


def states(mesh, p, oracle, iters):
    """A free stream along x with tiny cross-stream momenta in half of its
    cells, and the oracle's state after the iterations."""
    x, y, tri = mesh.nodes()
    c = oracle.Case(x, y, tri, oracle.params_from_e2d(p))
    w = c.state()
    rng = np.random.default_rng(8)
    w[:, 2] = rng.choice([0.0, 1e-310, -3e-312, 5e-324], len(w), p=[0.5, 0.2, 0.2, 0.1])
    c.set_state(w)
    c.run(iters)
    assert np.all(np.isfinite(c.state()))
    return w, c.state()


def params(kw):
    return e2d.default_params(ma=0.5, alpha_deg=0.0, cfl=1.0, **kw)


@pytest.mark.parametrize("iters", [1, 4])
@pytest.mark.parametrize("kw", KW)
@pytest.mark.parametrize("ni,nj", [(33, 9), (101, 60), (157, 77), (251, 201)])  # tiles; the face list with 4, 2, 1 threads
def test_solver(lib, oracle, ni, nj, kw, iters):
    mesh, p = e2d.Mesh.ogrid(ni, nj, seed=5), params(kw)
    w, ref = states(mesh, p, oracle, iters)
    s = e2d.Solver(mesh, p)
    s.set_state(w)
    s.step(iters)
    assert np.array_equal(s.state(), ref)


@pytest.mark.parametrize("kw", KW)
@pytest.mark.parametrize("sizes", [((33, 9), (40, 12)), ((101, 60), (33, 9))])  # tiles, the face list
def test_batch(lib, oracle, sizes, kw):
    meshes, p = [e2d.Mesh.ogrid(*s, seed=5) for s in sizes], params(kw)
    b = e2d.Batch(meshes, [p] * len(meshes))
    refs = [states(m, p, oracle, 3) for m in meshes]
    for c, (w, _) in enumerate(refs):
        b.set_state(c, w)
    b.step(3)
    for c, (_, ref) in enumerate(refs):
        assert np.array_equal(b.state(c), ref), c


@pytest.mark.parametrize("kw", KW)
@pytest.mark.parametrize("ni,nj", [(33, 9), (101, 60)])  # tiles with 4 and 2 threads a cell
def test_allocation_free(lib, oracle, ni, nj, kw):
    import torch
    mesh, p = e2d.Mesh.ogrid(ni, nj, seed=5), params(kw)
    w, ref = states(mesh, p, oracle, 3)
    dev = [torch.from_numpy(a).cuda() for a in (*file_order_layout(mesh), w.ravel().copy(), np.zeros(3))]
    topo, S, R, area, state, res = (ctypes.c_void_p(t.data_ptr()) for t in dev)
    epsm = ctypes.c_double(0.0)
    _lib.check(lib.e2d_step_noalloc(len(w), topo, S, R, area, ctypes.byref(p), 3, state, res, ctypes.byref(epsm), None))
    assert np.array_equal(dev[4].cpu().numpy().reshape(-1, 4), ref)
