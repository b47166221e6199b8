"""Which FP32 meshes run whole iterations in one launch: up to 16384 cells, but
above 12288 not with less than two smoothing sweeps and more than three stages,
where the launches of the passes are faster.  Both sides of the line against
the passes (a block size other than the default takes those), bit for bit."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu

R = [0.1, 0.15, 0.2, 0.3, 0.4, 0.5, 0.7, 1.0]


@pytest.mark.parametrize("ni,nj,stages,sweeps,launches", [
    (128, 48, 8, 0, 1), (150, 41, 3, 0, 1), (150, 41, 4, 0, 13), (150, 41, 4, 1, 13), (150, 41, 4, 2, 1),
    (128, 64, 8, 1, 25), (128, 64, 3, 1, 1), (128, 64, 8, 3, 1), (128, 65, 4, 2, 17)])
def test_line(lib, ni, nj, stages, sweeps, launches):
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    kw = dict(ma=0.5, alpha_deg=1.0, cfl=0.1, precision=e2d.E2D_FP32, rk_stages=stages, rk_coef=R[8 - stages:],
              irs_sweeps=sweeps)
    a = e2d.Solver(mesh, e2d.default_params(**kw))
    b = e2d.Solver(mesh, e2d.default_params(**kw, block_size=64))
    for s in (a, b):
        s.step(1)
        s.step(6)
    assert a.launches_per_iteration() == launches
    assert np.array_equal(a.state(), b.state())


@pytest.mark.parametrize("ni,nj", [(128, 48), (150, 41), (128, 64)])
def test_single_iterations(lib, ni, nj):
    """A call of one iteration takes the passes above 12288 cells; calls of one and
    of several iterations mix freely, over a growth of the history too."""
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    kw = dict(ma=0.5, alpha_deg=1.0, cfl=0.5, precision=e2d.E2D_FP32)
    a = e2d.Solver(mesh, e2d.default_params(**kw))
    b = e2d.Solver(mesh, e2d.default_params(**kw, block_size=64))
    for n in (1, 1, 3, 1, 2, 1, 1100, 1):
        a.step(n)
        b.step(n)
    assert np.array_equal(a.state(), b.state())
    np.testing.assert_allclose(a.history(), b.history(), rtol=1e-9)  # sums to about 48 bits, grouped otherwise
