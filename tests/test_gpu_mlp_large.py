"""Training with more batch tiles than SMs, where a CTA of the chains carries two
tiles, some CTAs a third one alone, and large networks run their weight gradients
layer by layer on two streams with shared partials: gradients and losses
against the per-tile kernels (E2D_MLP_WS=0), and steps repeated bit for bit.

Tolerances: both sides round the same quantities to BF16 (2^-9 of a value), the
sums before the rounding differ in FP32 order only, so a few roundings go the
other way: far below sqrt(layers) 2^-9 of a gradient's norm (0.6 % at eight)."""
import os

import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu


def rows(n):
    rng = np.random.default_rng(9)
    x = np.zeros((n, 32), np.float32)
    x[:, :22] = rng.normal(size=(n, 22))
    return x, (rng.normal(size=(n, 4)) * 0.3).astype(np.float32)


def on_both(call):
    out = []
    for mode in ("1", "0"):
        os.environ["E2D_MLP_WS"] = mode
        try:
            out.append(call())
        finally:
            os.environ.pop("E2D_MLP_WS", None)
    return out


@pytest.mark.parametrize("batch", [18432, 20480, 40960, 65536])  # 144, 160, 320 and 512 tiles
@pytest.mark.parametrize("layers", [1, 3, 5, 8])
def test_gradient(lib, batch, layers):
    x, t = rows(batch)
    (l1, g1), (l0, g0) = on_both(lambda: e2d.MLP(nhidden=layers, batch=batch, seed=4).gradient(x, t))
    assert abs(l1 - l0) <= 1e-3 * abs(l0)
    off = 0
    for l in range(layers + 1):  # tensor by tensor: a wrong layer does not hide in the whole
        r, c = (4 if l == layers else 256), (32 if l == 0 else 256)
        for size in (r * c, r):
            a, b = g1[off:off + size].astype(np.float64), g0[off:off + size].astype(np.float64)
            off += size
            assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), (l, size)
    assert off == len(g1)


@pytest.mark.parametrize("batch,layers", [(20480, 3), (20480, 8), (40960, 5), (65536, 5)])
def test_training(lib, batch, layers):
    x, t = rows(50000)

    def train():
        net = e2d.MLP(nhidden=layers, batch=batch, seed=4, lr=1e-4)
        net.set_data(x, t)
        return net.train(4), net.params(), net.forward(x[:3000])

    (l1, p1, y1), (l0, p0, y0) = on_both(train)
    assert np.all(np.abs(l1 - l0) <= 1e-2 * l0)
    l2, p2, y2 = train()
    assert np.array_equal(l1, l2) and np.array_equal(p1, p2) and np.array_equal(y1, y2)
    # four Adam steps move a parameter by 4 lr at most, whatever its gradient's sign
    assert np.max(np.abs(p1 - p0)) <= 8.1e-4
