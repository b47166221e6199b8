"""Features and wall distances computed on the GPU, against the same in numpy
FP64 (every wall face of every cell), and predictions for row counts around
the tile sizes, against the rows of one large call."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj", [(16, 4), (33, 7), (96, 24)])  # wall faces: one box of 16, a remainder, several
def test_features_against_numpy(lib, ni, nj):
    mesh = e2d.Mesh.ogrid(ni, nj, seed=3)
    f = e2d.MLP.features(mesh, 0.6, 1.5).astype(np.float64)
    x, y, tri = mesh.nodes()
    cx, cy = x[tri - 1].mean(1), y[tri - 1].mean(1)
    ei, _, _, _ = mesh.topology()
    w = ei[ei[:, 0] == 2][:, 5:7] - 1
    a = np.stack([x[w[:, 0]], y[w[:, 0]]], 1)
    e = np.stack([x[w[:, 1]], y[w[:, 1]]], 1) - a
    p = np.stack([cx, cy], 1)[:, None] - a
    t = np.clip((p * e).sum(-1) / (e * e).sum(-1), 0.0, 1.0)
    d = np.sqrt(((p - t[..., None] * e) ** 2).sum(-1).min(1))
    # FP32 values: half a unit in the last place is 6e-8 of the value
    for k, ref in ((0, cx), (1, cy), (2, np.log(d + 1e-3))):
        assert np.all(np.abs(f[:, k] - ref) <= 1e-7 * np.abs(ref) + 1e-12), k
    assert np.all(f[:, 3] == np.float32(0.6)) and np.all(f[:, 22:] == 0.0)
    assert np.allclose(f[:, 6:22:2] ** 2 + f[:, 7:22:2] ** 2, 1.0, rtol=0, atol=3e-7)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 256, 257, 2047, 2048, 2049, 4100])
def test_prediction_rows_do_not_depend_on_the_call(lib, n):
    net = e2d.MLP(nhidden=2, batch=2048, seed=5)
    rng = np.random.default_rng(n)
    x = np.zeros((6144, 32), np.float32)
    x[:, :22] = rng.normal(size=(6144, 22))
    assert np.array_equal(net.forward(x[:n]), net.forward(x)[:n])
