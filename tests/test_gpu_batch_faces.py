"""FP64 batches above 12000 cells in all, whose passes A and B work from a list of
the faces of every case: each case keeps the bits of its own single-case run
(of fewer cells, in tiles), with padding, options, halted cases and every block
size."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu

SIZES = [(64, 48, 1), (50, 33, 2), (80, 41, 3)]  # 6144, 3300 and 6560 cells


def compare(sizes, iters, block=128, solve=False, **kw):
    meshes = [e2d.Mesh.ogrid(ni, nj, seed=s) for ni, nj, s in sizes]
    params = [e2d.default_params(ma=m, alpha_deg=1.0, cfl=1.2, ordering=e2d.E2D_ORDER_MORTON, maxstep=400,
                                 block_size=block, **kw) for m in (0.5, 0.62, 0.4)[:len(sizes)]]
    singles = [e2d.Solver(m, p) for m, p in zip(meshes, params)]
    b = e2d.Batch(meshes, params)
    b.set_launch(block, 0)
    b.step(iters)
    for s in singles:
        s.step(iters)
    if solve:  # the first case halts, the others go on
        epsl = singles[0].history()[-1] * (1 + 1e-12)
        b.solve(6, epsl)
        for s in singles:
            s.solve(6, epsl)
    for c, s in enumerate(singles):
        assert np.array_equal(b.state(c), s.state()), c
        assert np.array_equal(b.history(c), s.history()), c
    return b


@pytest.mark.parametrize("block", [32, 128, 256])
def test_blocks(lib, block):
    b = compare(SIZES, 5, block, solve=True)
    assert b.launches_per_iteration() == 21


@pytest.mark.parametrize("kw", [dict(limiter=1), dict(limiter=3, limiter_freeze=2), dict(positivity_fix=1),
                                dict(global_dt=1), dict(first_order_iters=2)])
def test_options(lib, kw):
    compare(SIZES, 5, **kw)


def test_large(lib):  # one thread per cell in pass A
    compare([(251, 200, 1), (50, 33, 2)], 3)


def test_line(lib):
    assert compare(SIZES[:1] + [(50, 55, 2)], 3).launches_per_iteration() == 17  # 6144 + 5632 with padding
