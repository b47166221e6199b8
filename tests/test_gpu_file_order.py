"""The kernels chosen by size, in file order (the library's default) and in
reverse Cuthill-McKee order, where a face's two cells lie far apart in memory or
a tile shares few faces: FP64 against the CPU oracle bit for bit, FP32 small
meshes against the passes, batches against their single cases."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu

ORDERS = [e2d.E2D_ORDER_FILE, e2d.E2D_ORDER_RCM]
KW = dict(ma=0.6, alpha_deg=1.5, cfl=1.2)


@pytest.mark.parametrize("ordering", ORDERS)
@pytest.mark.parametrize("ni,nj", [(77, 77), (101, 60), (157, 77), (251, 201)])  # tiles; a list with 4, 2 and 1 threads a cell
@pytest.mark.parametrize("kw", [{}, dict(limiter=3, limiter_freeze=2)])
def test_fp64(lib, oracle, ordering, ni, nj, kw):
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    p = e2d.default_params(**KW, ordering=ordering, **kw)
    s = e2d.Solver(mesh, p)
    s.step(3)
    x, y, tri = mesh.nodes()
    c = oracle.Case(x, y, tri, oracle.params_from_e2d(p))
    c.run(3)
    assert np.array_equal(s.state(), c.state())


@pytest.mark.parametrize("ordering", ORDERS)
@pytest.mark.parametrize("ni,nj,kw", [(8, 1, {}), (65, 16, {}), (129, 32, {}), (128, 64, {}), (128, 32, dict(limiter=2))])
def test_fp32_small(lib, ordering, ni, nj, kw):
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    kw = dict(**KW, precision=e2d.E2D_FP32, ordering=ordering, **kw)
    a = e2d.Solver(mesh, e2d.default_params(**kw))
    b = e2d.Solver(mesh, e2d.default_params(**kw, block_size=64))
    assert a.launches_per_iteration() == 1 and b.launches_per_iteration() == 17
    for n in (1, 9):
        a.step(n)
        b.step(n)
    assert np.array_equal(a.state(), b.state())


@pytest.mark.parametrize("ordering", ORDERS)
@pytest.mark.parametrize("precision", [e2d.E2D_FP64, e2d.E2D_FP32])
def test_batches(lib, ordering, precision):
    meshes = [e2d.Mesh.ogrid(ni, nj, seed=s) for ni, nj, s in ((64, 48, 1), (50, 33, 2), (80, 41, 3))]
    params = [e2d.default_params(ma=m, cfl=1.2, ordering=ordering, precision=precision) for m in (0.5, 0.62, 0.4)]
    b = e2d.Batch(meshes, params)
    b.step(5)
    for c, (m, p) in enumerate(zip(meshes, params)):
        s = e2d.Solver(m, p)
        s.step(5)
        assert np.array_equal(b.state(c), s.state()), c
