"""A network's, a solver's and a batch's first calls while the legacy default
stream has work of the caller pending: they read buffers on streams of their
own, which do not wait for the default one.  Results against the same calls
with the default stream idle, bit for bit."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu


def pending():
    """Queues some tens of milliseconds of work on the default stream."""
    import torch
    a = torch.ones(4096, 4096, device="cuda")
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    for _ in range(40):
        torch.mm(a, a, out=b)
    return b


def rows(n):
    rng = np.random.default_rng(6)
    x = np.zeros((n, 32), np.float32)
    x[:, :22] = rng.normal(size=(n, 22))
    return x, rng.normal(size=(n, 4)).astype(np.float32)


def first_gradient(net):
    loss, g = net.gradient(*rows(4096))
    return np.append(g, np.float32(loss))


def first_training(net):
    net.set_data(*rows(20000))
    net.train(3)
    return net.params()


def copied_params(net):
    net.set_params(net.params()[::-1].copy())
    return net.forward(rows(300)[0])


@pytest.mark.parametrize("call", [first_gradient, first_training, copied_params, lambda net: net.forward(rows(5000)[0])])
@pytest.mark.parametrize("made_before", [True, False])
def test_first_calls_of_a_network(lib, call, made_before):
    ref = call(e2d.MLP(nhidden=3, batch=4096, seed=4))
    assert np.all(np.isfinite(ref)) and np.any(ref != 0)
    net = e2d.MLP(nhidden=3, batch=4096, seed=4) if made_before else None
    work = pending()
    got = call(net or e2d.MLP(nhidden=3, batch=4096, seed=4))
    assert np.array_equal(got, ref)
    del work


def solver_state(precision):
    s = e2d.Solver(e2d.Mesh.ogrid(70, 40, seed=2), e2d.default_params(ma=0.6, cfl=1.2, precision=precision, block_size=64))
    s.step(2)
    if precision == e2d.E2D_FP32:
        s.set_precision(e2d.E2D_FP64)
        s.step(2)
    return s.state()


def batch_state(precision):
    b = e2d.Batch([e2d.Mesh.ogrid(40, 9, seed=2), e2d.Mesh.ogrid(33, 20, seed=1)],
                  [e2d.default_params(ma=m, cfl=1.2, precision=precision) for m in (0.5, 0.6)])
    b.step(2)
    b.set_launch(64, 8)
    b.step(2)
    return np.concatenate([b.state(0), b.state(1)])


@pytest.mark.parametrize("call", [solver_state, batch_state])
@pytest.mark.parametrize("precision", [e2d.E2D_FP32, e2d.E2D_FP64])
def test_first_steps(lib, call, precision):
    ref = call(precision)
    work = pending()
    assert np.array_equal(call(precision), ref)
    del work


def test_features_of_many_wall_faces(lib):
    """4096 wall faces: the copies of their segments and boxes are over the
    64 KB that a copy from pageable memory takes at once."""
    mesh = e2d.Mesh.ogrid(4096, 2, seed=3)
    x, y, tri = mesh.nodes()
    ei, _, _, _ = mesh.topology()
    w = ei[ei[:, 0] == 2][:, 5:7] - 1
    a = np.stack([x[w[:, 0]], y[w[:, 0]]], 1)
    e = np.stack([x[w[:, 1]], y[w[:, 1]]], 1) - a
    c = np.stack([x[tri - 1].mean(1), y[tri - 1].mean(1)], 1)
    assert len(w) == 4096
    work = pending()
    f = e2d.MLP.features(mesh, 0.6, 1.5).astype(np.float64)
    for k in range(0, len(c), 1000):
        p = c[k:k + 1000, None] - a
        t = np.clip((p * e).sum(-1) / (e * e).sum(-1), 0.0, 1.0)
        ref = np.log(np.sqrt(((p - t[..., None] * e) ** 2).sum(-1).min(1)) + 1e-3)
        # FP32 values: half a unit in the last place is 6e-8 of the value
        assert np.all(np.abs(f[k:k + 1000, 2] - ref) <= 1e-7 * np.abs(ref) + 1e-12)
    del work
