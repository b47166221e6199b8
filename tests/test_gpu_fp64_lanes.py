"""FP64 passes A and B with several threads per cell (small meshes take four
and two, larger ones two and one), against the CPU oracle, bit for bit: sizes on
both sides of each change of shape, partial tiles, block sizes from the smallest
to the largest, and the options that pass A carries."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu


def run(oracle, ni, nj, iters, **kw):
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    p = e2d.default_params(ma=0.6, alpha_deg=1.5, cfl=1.2, ordering=e2d.E2D_ORDER_MORTON, **kw)
    s = e2d.Solver(mesh, p)
    s.step(iters)
    x, y, tri = mesh.nodes()
    pf = e2d.default_params(ma=0.6, alpha_deg=1.5, cfl=1.2, **kw)
    c = oracle.Case(x, y, tri, oracle.params_from_e2d(pf))
    c.run(iters)
    assert np.array_equal(s.state(), c.state())


@pytest.mark.parametrize("ni,nj", [(9, 3), (77, 77), (78, 77), (150, 133), (151, 134)])  # around 12000 and 40000 cells
def test_sizes(lib, oracle, ni, nj):
    run(oracle, ni, nj, 3)


@pytest.mark.parametrize("block", [32, 96, 256])
def test_blocks(lib, oracle, block):
    run(oracle, 33, 9, 4, block_size=block)


@pytest.mark.parametrize("kw", [dict(limiter=1), dict(limiter=2), dict(limiter=3, limiter_freeze=2),
                                dict(positivity_fix=1), dict(global_dt=1), dict(first_order_iters=2)])
def test_options(lib, oracle, kw):
    run(oracle, 33, 9, 5, **kw)
