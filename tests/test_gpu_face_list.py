"""FP64 meshes above 12000 cells, whose passes A and B work from a list of the
faces, against the CPU oracle, bit for bit: both sides of the line and
of the changes of threads per cell, block sizes from the smallest to the largest,
and the options."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu


def run(oracle, ni, nj, iters, **kw):
    mesh = e2d.Mesh.ogrid(ni, nj, seed=5)
    s = e2d.Solver(mesh, e2d.default_params(ma=0.6, alpha_deg=1.5, cfl=1.2, ordering=e2d.E2D_ORDER_MORTON, **kw))
    s.step(iters)
    x, y, tri = mesh.nodes()
    kw.pop("block_size", None)
    c = oracle.Case(x, y, tri, oracle.params_from_e2d(e2d.default_params(ma=0.6, alpha_deg=1.5, cfl=1.2, **kw)))
    c.run(iters)
    assert np.array_equal(s.state(), c.state())
    return s


@pytest.mark.parametrize("ni,nj,launches", [(100, 60, 17), (101, 60, 21), (157, 77, 21), (251, 200, 21)])
def test_line(lib, oracle, ni, nj, launches):
    assert run(oracle, ni, nj, 3).launches_per_iteration() == launches


@pytest.mark.parametrize("ni", [101, 157])
@pytest.mark.parametrize("kw", [dict(block_size=32), dict(block_size=256), dict(limiter=1), dict(limiter=2),
                                dict(limiter=3, limiter_freeze=2), dict(positivity_fix=1), dict(global_dt=1),
                                dict(first_order_iters=2)])
def test_options(lib, oracle, kw, ni):
    run(oracle, ni, 77, 4, **kw)
