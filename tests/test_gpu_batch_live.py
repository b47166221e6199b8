"""Cases of a batch that halt and are taken up again: the table of live chunks
follows the cases' halt flags, whatever the block size, and every case keeps the
bits of its own single-case run."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [32, 128, 256])
@pytest.mark.parametrize("prec", [e2d.E2D_FP64, e2d.E2D_FP32])
def test_halted_cases_go_on(lib, prec, block):
    sizes = [(32, 8, 1), (48, 11, 2), (64, 16, 3), (21, 6, 5)]  # 21 x 6: less than a chunk
    meshes = [e2d.Mesh.ogrid(ni, nj, seed=s) for ni, nj, s in sizes]
    params = [e2d.default_params(ma=m, alpha_deg=1.0, cfl=1.2, precision=prec, ordering=e2d.E2D_ORDER_MORTON,
                                 maxstep=400, block_size=block) for m in (0.5, 0.6, 0.4, 0.7)]
    singles = [e2d.Solver(m, p) for m, p in zip(meshes, params)]
    for s in singles:
        s.step(60)
    epsl = float(np.median([s.history()[30] for s in singles]))
    singles = [e2d.Solver(m, p) for m, p in zip(meshes, params)]
    b = e2d.Batch(meshes, params)
    b.set_launch(block, 0)
    n = b.solve(60, epsl)
    for s in singles:
        s.solve(60, epsl)
    assert len(set(n)) > 1
    for k in range(2):  # some cases halted, then all run again
        for c, s in enumerate(singles):
            assert np.array_equal(b.state(c), s.state()), (k, c)
            assert np.array_equal(b.history(c), s.history()), (k, c)
        if k == 0:
            b.step(9)
            for s in singles:
                s.step(9)
