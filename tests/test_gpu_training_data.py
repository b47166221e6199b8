"""e2d_mlp_set_data takes any batch size (the batch is checked where it is used)
and row counts around the pieces it is uploaded in; a call that fails leaves
no data behind, and the next one works."""
import ctypes

import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d
from gpueularsolver2d_gb300._lib import E2DError

pytestmark = pytest.mark.gpu


def rows(n):
    rng = np.random.default_rng(n)
    x = np.zeros((n, 32), np.float32)
    x[:, :22] = rng.normal(size=(n, 22))
    return x, rng.normal(size=(n, 4)).astype(np.float32)


@pytest.mark.parametrize("batch", [0, -4096, 1000])
def test_batch_is_checked_where_it_is_used(lib, batch):
    net = e2d.MLP(nhidden=1, batch=batch)
    net.set_data(*rows(3000))
    if batch:
        with pytest.raises(E2DError, match="multiple of 2048"):
            net.train(1)


def batch_rows(seed, step, batch, n):
    """The rows that training step `step` (from 1) draws (k_gather)."""
    j = np.arange(batch, dtype=np.uint64)
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9e3779b97f4a7c15) * (np.uint64(step * 1315423911) + j + np.uint64(1))
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
    return ((z ^ (z >> np.uint64(31))) % np.uint64(n)).astype(np.int64)


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 5000])  # uploaded in pieces of 2048 rows
def test_every_row_arrives(lib, n):
    net = e2d.MLP(nhidden=1, batch=2048, seed=7)
    x, t = rows(n)
    net.set_data(x, t)
    i = batch_rows(7, 1, 2048, n)
    y = net.forward(x[i]).astype(np.float64)
    # the same FP32 outputs but for the order of a sum of 256 terms (2^-24 each)
    assert net.train(1)[0] == pytest.approx(np.mean((y - t[i]) ** 2), rel=1e-5)


def test_prediction_in_several_pieces(lib):  # of 65536 rows
    x = rows(140000)[0]
    y = e2d.MLP(nhidden=1, batch=2048).forward(x)
    assert np.array_equal(e2d.MLP(nhidden=1, batch=262144).forward(x), y)


def test_a_failed_call_leaves_no_data(lib):
    net = e2d.MLP(nhidden=1, batch=2048)
    x, t = rows(4096)
    net.set_data(x, t)
    net.train(1)
    fp = ctypes.POINTER(ctypes.c_float)
    assert lib.e2d_mlp_set_data(net._h, 1 << 50, x.ctypes.data_as(fp), t.ctypes.data_as(fp)) != 0
    with pytest.raises(E2DError, match="no training data"):
        net.train(1)
    net.set_data(x, t)
    assert np.isfinite(net.train(1)[0])


def test_a_batch_that_does_not_fit_stays_refused(lib):
    """The first call's error is every later call's: none runs on a part of the
    buffers.  (The first hidden layer would take 256 GB.)"""
    net = e2d.MLP(nhidden=1, batch=2 ** 29)
    for _ in range(2):
        with pytest.raises(E2DError, match="out of memory"):
            net.forward(rows(1)[0])
    net.close()
    assert np.all(np.isfinite(e2d.MLP(nhidden=1, batch=2048).forward(rows(1)[0])))
