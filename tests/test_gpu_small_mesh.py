"""FP32 meshes small enough for one launch to run whole iterations (one cluster
holds the mesh) against the pass-by-pass kernels (a block size other than the
default takes those): states bit for bit, and with them the residuals but for
the grouping of their partial sums.  Against a batch of one, which groups as
the default block does, the residuals are the same bits too.  Sizes: fewer cells
than CTAs, one or two cells to a thread, partial groups of 128, the largest."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu

KW = dict(ma=0.6, alpha_deg=1.5, cfl=1.2, precision=e2d.E2D_FP32, ordering=e2d.E2D_ORDER_MORTON, maxstep=2000)


def compare(ni, nj, iters, **kw):
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    kw = {**KW, **kw}
    a = e2d.Solver(mesh, e2d.default_params(**kw))
    b = e2d.Batch([mesh], [e2d.default_params(**kw)])
    c = e2d.Solver(mesh, e2d.default_params(**kw, block_size=64))
    for n in iters:
        a.step(n)
        b.step(n)
        c.step(n)
    assert np.array_equal(a.state(), b.state(0)) and np.array_equal(a.history(), b.history(0))
    assert np.array_equal(a.state(), c.state())
    np.testing.assert_allclose(a.history(), c.history(), rtol=1e-9)  # sums to about 48 bits, grouped otherwise


@pytest.mark.parametrize("ni,nj", [(8, 1), (9, 7), (64, 16), (65, 16), (128, 32), (129, 32), (150, 41), (128, 64)])
def test_sizes(lib, ni, nj):
    compare(ni, nj, [1, 12])


@pytest.mark.parametrize("kw", [dict(irs_sweeps=0), dict(irs_sweeps=1), dict(irs_sweeps=3), dict(rk_stages=1, rk_coef=[0.4]),
                                dict(limiter=1), dict(limiter=3, limiter_freeze=3), dict(limiter_freeze_resd=0.9),
                                dict(positivity_fix=1), dict(first_order_iters=4), dict(global_dt=1)])
def test_options(lib, kw):
    compare(33, 9, [2, 9], **{**dict(cfl=0.6), **kw})


def test_stops_at_the_residual(lib):
    """The launch stops by itself where the passes stop, also over the
    boundary of a launch's iterations, and a stopped solver goes on."""
    mesh = e2d.Mesh.ogrid(64, 16, seed=2)
    a = e2d.Solver(mesh, e2d.default_params(**KW))
    b = e2d.Solver(mesh, e2d.default_params(**KW, block_size=64))
    for epsl in (0.5, 0.2, 0.05):
        ha, hb = a.solve(900, epsl), b.solve(900, epsl)
        assert len(ha) == len(hb) and np.array_equal(a.state(), b.state())
    a.step(300)
    b.step(300)
    assert np.array_equal(a.state(), b.state())


def test_profiled_passes_advance_like_steps(lib):
    """e2d_profile_passes launches the passes one by one whatever the mesh."""
    mesh = e2d.Mesh.ogrid(64, 16, seed=2)
    a = e2d.Solver(mesh, e2d.default_params(**KW))
    b = e2d.Solver(mesh, e2d.default_params(**KW))
    ms, launches = a.profile_passes(5)
    b.step(5)
    assert launches.tolist() == [20, 20, 20, 20, 5] and np.all(ms > 0)
    assert np.array_equal(a.state(), b.state()) and np.array_equal(a.history(), b.history())
