"""The work that a user of this framework has it do, as a set of cases.

A solver case is one run from a given state: the state goes in, a number of
iterations run, the state, the residuals and the lift / drag come out.  A batch
case is the same for many cases advanced together.  The network cases are the
learned warm start: training steps, the gradient of one batch, and the
prediction of a state for a new condition (features of every cell of the mesh,
then the network).

Meshes are O-grids around NACA 0012 (chord 1, radius 20, first wall spacing
2e-3, random diagonals, 5 % jitter); the states are a subsonic flow that has
developed around the profile, not the free stream.
"""
import math

import numpy as np
import torch

import gpueularsolver2d_gb300 as e2d

RK4 = [0.0833, 0.2069, 0.4265, 1.0]
RK5 = [0.0695, 0.1602, 0.2898, 0.5060, 1.0]
GAMMA = 1.4
WALL_BOX = 2.0
MAXSTEP = 60000  # residual history that a run may need


def listed():
    return [
        # smallest call: the default parameters of the library (FP64, cells in file order) on a first
        # mesh, as the reference's own program is used
        dict(name="solve_fp64_2k", kind="solve", ni=64, nj=16, fp64=True, order=0, stages=4, ma=0.5, alpha=1.25,
             cfl=1.5, irs_eps=0.8, sweeps=2, limiter=0, k=5.0, frozen=False, iters=100),
        # the small-mesh configuration: FP32, five stages, no smoothing needed
        dict(name="solve_fp32_8k", kind="solve", ni=128, nj=32, fp64=False, order=1, stages=5, ma=0.5, alpha=1.25,
             cfl=2.0, irs_eps=0.6, sweeps=2, limiter=0, k=5.0, frozen=False, iters=200),
        # the FP64 tail of a converged run (limiter values frozen), most of the wall time of a 1e-6 drop
        dict(name="tail_fp64_34k", kind="solve", ni=251, nj=67, fp64=True, order=1, stages=4, ma=0.65, alpha=1.0,
             cfl=2.0, irs_eps=0.8, sweeps=2, limiter=3, k=5.0, frozen=True, iters=50),
        # the transonic configuration in FP32 with the limiter that converges
        dict(name="solve_fp32_131k", kind="solve", ni=512, nj=128, fp64=False, order=1, stages=4, ma=0.80, alpha=1.25,
             cfl=2.0, irs_eps=0.6, sweeps=2, limiter=3, k=5.0, frozen=False, iters=100),
        # the plain FP64 solver on a fine mesh, the run that FP32 results are held against
        dict(name="solve_fp64_1m", kind="solve", ni=1024, nj=512, fp64=True, order=1, stages=4, ma=0.78, alpha=2.0,
             cfl=2.0, irs_eps=0.8, sweeps=2, limiter=0, k=5.0, frozen=False, iters=10),
        # the large-mesh configuration, FP32
        dict(name="solve_fp32_4m", kind="solve", ni=2048, nj=1024, fp64=False, order=1, stages=4, ma=0.78, alpha=2.0,
             cfl=2.0, irs_eps=0.8, sweeps=2, limiter=0, k=5.0, frozen=False, iters=100),
        # sweep of uneven cases (64..512 around, 16..128 out), each its own mesh and condition
        dict(name="sweep_fp32_60", kind="batch", ncase=60, ni=512, nj=128, uneven=True, fp64=False, order=1, stages=4,
             ma=0.3, ma1=0.85, cfl=2.0, irs_eps=0.8, sweeps=2, limiter=0, k=5.0, iters=50),
        # training data of the warm start: many conditions on one mesh, smooth limiter, values kept for freezing
        dict(name="generate_fp32_24", kind="batch", ncase=24, ni=256, nj=64, uneven=False, fp64=False, order=1,
             stages=4, ma=0.575, ma1=0.70, cfl=2.0, irs_eps=0.8, sweeps=2, limiter=1, k=10.0, iters=50),
        # training: the configured network and batch; a small batch of a deeper network
        dict(name="train_64k", kind="train", nhidden=5, batch=65536, samples=500000, steps=10),
        dict(name="train_4k", kind="train", nhidden=8, batch=4096, samples=70001, steps=20),
        # gradient of one given batch (checks of the training, optimisers of the user's own)
        dict(name="gradient_16k", kind="gradient", nhidden=5, batch=16384),
        # the prediction for a new condition on a mesh: features of every cell and the network
        dict(name="predict_34k", kind="predict", ni=251, nj=67, nhidden=5, batch=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "train", "gradient", "predict"])
    if kind == "solve":
        fp64 = rng.random() < 0.5
        limiter = rng.choice([0, 0, 1, 3])
        sweeps = rng.choice([0, 2, 2, 2, 3])  # a single sweep is not stable with this scheme
        cells = _log(rng, 2000, 1000000 if fp64 else 4000000)
        ni = max(48, int(round(math.sqrt(cells) * rng.uniform(0.8, 1.7))))
        nj = max(12, cells // (2 * ni))
        return dict(kind=kind, ni=ni, nj=nj, fp64=fp64, order=rng.choice([0, 1, 1, 1, 2]), stages=rng.choice([4, 4, 5]),
                    ma=rng.uniform(0.4, 0.8), alpha=rng.uniform(-1.0, 3.0), cfl=rng.uniform(1.0, 2.0) if sweeps > 1 else rng.uniform(0.5, 1.0),
                    irs_eps=rng.choice([0.6, 0.8]), sweeps=sweeps, limiter=limiter,
                    k=rng.choice([5.0, 10.0]), frozen=limiter > 0 and rng.random() < 0.3,
                    iters=max(5, min(100, int((6e6 if fp64 else 3e8) / cells))))
    if kind == "batch":
        uneven = rng.random() < 0.6
        fp64 = rng.random() < 0.25
        return dict(kind=kind, ncase=_log(rng, 3, 12 if fp64 else 60), ni=_log(rng, 96, 512), nj=_log(rng, 24, 100),
                    uneven=uneven, fp64=fp64, order=rng.choice([0, 1, 1, 2]), stages=4, ma=0.4, ma1=0.8,
                    cfl=rng.uniform(1.0, 2.0), irs_eps=0.8, sweeps=2, limiter=rng.choice([0, 1, 3]), k=10.0,
                    iters=10 if fp64 else 40)
    if kind == "train":
        return dict(kind=kind, nhidden=rng.randint(2, 8), batch=2048 * _log(rng, 1, 32), samples=_log(rng, 30000, 500000),
                    steps=rng.randint(5, 20))
    if kind == "gradient":
        return dict(kind=kind, nhidden=rng.randint(1, 8), batch=2048 * _log(rng, 1, 16))
    return dict(kind=kind, ni=_log(rng, 64, 512), nj=_log(rng, 16, 256), nhidden=rng.randint(3, 8), batch=65536)


# ---- inputs -----------------------------------------------------------------

def _mesh(ni, nj, seed):
    """Nodes x, y and triangles (1-based, counter-clockwise) of a jittered O-grid."""
    rng = np.random.default_rng(seed)
    lo, hi = 1.0001, 40.0
    for _ in range(80):  # growth of the layers from 2e-3 to radius 20
        q = 0.5 * (lo + hi)
        if nj * math.log(q) > 30.0 or 2e-3 * (q ** nj - 1.0) / (q - 1.0) > 20.0:
            hi = q
        else:
            lo = q
    s = (q ** np.arange(nj + 1) - 1.0) / (q ** nj - 1.0)
    th = 2.0 * np.pi * (np.arange(ni)[None, :] + np.zeros((nj + 1, 1))) / ni
    s = np.repeat(s[:, None], ni, 1)
    jit = 0.05 * rng.uniform(-1.0, 1.0, (2, nj - 1, ni))
    th[1:-1] += jit[0] * 2.0 * np.pi / ni
    s[1:-1] += jit[1] * np.minimum(s[1:-1] - s[:-2], s[2:] - s[1:-1])
    c = 0.5 * (1.0 + np.cos(th))
    t = 0.6 * (0.2969 * np.sqrt(c) - 0.126 * c - 0.3516 * c ** 2 + 0.2843 * c ** 3 - 0.1036 * c ** 4)
    yw = np.where(np.sin(th) >= 0.0, t, -t)
    x = c + s * (0.5 + 20.0 * np.cos(th) - c)
    y = yw + s * (20.0 * np.sin(th) - yw)
    j, i = np.meshgrid(np.arange(nj), np.arange(ni), indexing="ij")
    a = j * ni + i + 1
    d = j * ni + (i + 1) % ni + 1
    b, c4 = a + ni, d + ni
    flip = rng.random((nj, ni)) < 0.5
    t0 = np.where(flip[..., None], np.stack([a, b, d], -1), np.stack([a, b, c4], -1))
    t1 = np.where(flip[..., None], np.stack([b, c4, d], -1), np.stack([a, c4, d], -1))
    tri = np.stack([t0, t1], 2).reshape(-1, 3).astype(np.int32)
    return x.ravel(), y.ravel(), tri


def _state(x, y, tri, ma, alpha, seed):
    """A flow past the profile: the velocity is turned and slowed near the wall as past an ellipse, the
    pressure follows from the total enthalpy, every cell is disturbed by up to 1e-3."""
    rng = np.random.default_rng(seed + 1)
    cx, cy = x[tri - 1].mean(1), y[tri - 1].mean(1)
    a = alpha * math.pi / 180.0
    ca, sa = math.cos(a), math.sin(a)
    z = ((cx - 0.5) + 1j * cy)
    r2 = np.abs(z) ** 2 + 0.12
    zi = np.conj(z) / r2  # 1 / z, bounded at the origin
    v = (ca - 1j * sa) - 0.035 * (ca + 1j * sa) * zi * zi - 0.04j * zi
    u, w = v.real, -v.imag
    p_inf = 1.0 / (GAMMA * ma * ma)
    h_inf = GAMMA / (GAMMA - 1.0) * p_inf + 0.5
    tt = np.maximum((h_inf - 0.5 * (u * u + w * w)) / (h_inf - 0.5), 0.5)
    rho = tt ** (1.0 / (GAMMA - 1.0))
    p = p_inf * rho ** GAMMA
    e = 1e-3 * rng.uniform(-1.0, 1.0, (4, len(cx)))
    rho, u, w, p = rho * (1 + e[0]), u * (1 + e[1]), w * (1 + e[2]), p * (1 + e[3])
    return np.ascontiguousarray(np.stack([rho, rho * u, rho * w, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + w * w)], 1))


def _params(case, ma, alpha):
    rk = RK5 if case["stages"] == 5 else RK4
    return e2d.default_params(ma=ma, alpha_deg=alpha, cfl=case["cfl"], maxstep=MAXSTEP, rk_stages=case["stages"],
                              rk_coef=rk, irs_eps=case["irs_eps"], irs_sweeps=case["sweeps"],
                              precision=e2d.E2D_FP64 if case["fp64"] else e2d.E2D_FP32, ordering=case["order"],
                              limiter=case["limiter"], limiter_k=case["k"],
                              limiter_freeze=1 if case.get("frozen") else 0,
                              limiter_freeze_resd=1e-3 if case["kind"] == "batch" and case["limiter"] == 1 else 0.0)


def _batch(case, seed):
    """[(ni, nj, mesh seed, Mach, alpha)] of a batch; even batches share one mesh."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(case["ncase"])
    out = []
    for c in range(case["ncase"]):
        ni, nj = case["ni"], case["nj"]
        if case["uneven"]:  # the sizes belong to the case, the meshes and conditions to the seed
            ni = max(32, int(ni * sizes.choice([0.125, 0.25, 0.5, 1.0])))
            nj = max(8, int(nj * sizes.choice([0.125, 0.25, 0.5, 1.0])))
        out.append((ni, nj, seed + (c if case["uneven"] else 0), float(rng.uniform(case["ma"], case["ma1"])),
                    float(rng.uniform(-1.0, 3.0))))
    return out


def _weights(nhidden, seed):
    """Initial weights of the network, flat in the order W0, b0, W1, b1, ..."""
    rng = np.random.default_rng(seed)
    out = []
    for layer in range(nhidden + 1):
        rows, cols = (4 if layer == nhidden else 256), (32 if layer == 0 else 256)
        fan = 22 if layer == 0 else 256
        w = rng.standard_normal((rows, cols)) * math.sqrt((1.0 if layer == nhidden else 2.0) / fan)
        out += [w.ravel(), 0.05 * rng.standard_normal(rows)]
    return np.concatenate(out).astype(np.float32)


def _samples(n, seed):
    """Normalised features and targets: a smooth function of the features, as the flow is."""
    rng = np.random.default_rng(seed + 2)
    x = np.zeros((n, 32), np.float32)
    x[:, :6] = rng.standard_normal((n, 6), np.float32)
    ph = (x[:, :2] @ rng.standard_normal((2, 8)).astype(np.float32)) * np.float32(2.0 * math.pi)
    x[:, 6:22:2], x[:, 7:22:2] = np.sin(ph), np.cos(ph)
    t = np.tanh(x[:, :22] @ (0.5 * rng.standard_normal((22, 4))).astype(np.float32))
    return x, np.ascontiguousarray(t)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        x, y, tri = _mesh(case["ni"], case["nj"], seed)
        s = e2d.Solver(e2d.Mesh.from_arrays(x, y, tri), _params(case, case["ma"], case["alpha"]))
        w = _state(x, y, tri, case["ma"], case["alpha"], seed)
        if case["frozen"]:  # one iteration: the limiter values are frozen from here on
            s.set_state(w)
            s.step(1)
        return dict(kind=kind, case=case, solver=s, w=w)
    if kind == "batch":
        specs = _batch(case, seed)
        arrays = {q[:3]: _mesh(*q[:3]) for q in specs}
        meshes = {q: e2d.Mesh.from_arrays(*a) for q, a in arrays.items()}
        b = e2d.Batch([meshes[q[:3]] for q in specs], [_params(case, q[3], q[4]) for q in specs])
        w = [_state(*arrays[q[:3]], q[3], q[4], seed + c) for c, q in enumerate(specs)]
        return dict(kind=kind, case=case, batch=b, w=w)
    net = e2d.MLP(nhidden=case["nhidden"], batch=case["batch"], seed=3 + seed % 1000)
    net.set_params(_weights(case["nhidden"], seed))
    if kind == "train":
        net.set_data(*_samples(case["samples"], seed))
        return dict(kind=kind, case=case, net=net)
    if kind == "gradient":
        x, t = _samples(case["batch"], seed)
        return dict(kind=kind, case=case, net=net, x=x, t=t)
    mesh = e2d.Mesh.from_arrays(*_mesh(case["ni"], case["nj"], seed))
    mean, std = _normalisation()
    return dict(kind=kind, case=case, net=net, mesh=mesh, mean=mean, std=std)


def _normalisation():
    mean, std = np.zeros(32, np.float32), np.ones(32, np.float32)
    mean[:6] = [0.3, 0.0, -1.5, 0.65, 0.02, 1.0]
    std[:6] = [4.0, 4.0, 2.0, 0.09, 0.02, 0.001]
    return mean, std


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "solve":
        s = state["solver"]
        s.set_state(state["w"])
        resd = s.solve(case["iters"], 0.0)
        return {"state": s.state(), "resd": resd, "forces": np.array(s.forces())}
    if kind == "batch":
        b = state["batch"]
        n = case["ncase"]
        for c in range(n):
            b.set_state(c, state["w"][c])
        b.step(case["iters"])
        return {"states": [b.state(c) for c in range(n)],
                "forces": np.array([b.forces(c) for c in range(n)])}
    net = state["net"]
    if kind == "train":
        loss = net.train(case["steps"])
        return {"loss": loss, "params": net.params()}
    if kind == "gradient":
        loss, g = net.gradient(state["x"], state["t"])
        return {"loss": loss, "gradient": g}
    f = e2d.MLP.features(state["mesh"], 0.62, 1.1)
    y = net.forward((f - state["mean"]) / state["std"])
    return {"features": f, "prediction": y}


def work(case):
    """Per cell and stage of the solver: the state, the start state, the faces and their geometry are read
    once and the new state is written; roughly 750 operations.  A hidden layer of the network is 2 x 256 x 256
    operations a row and direction; its activation is kept for the way back."""
    kind = case["kind"]
    if kind in ("solve", "batch"):
        cells = 2 * case["ni"] * case["nj"]
        if kind == "batch":
            cells *= case["ncase"] * (0.2 if case["uneven"] else 1.0)
        size = 8 if case["fp64"] else 4
        n = cells * case["stages"] * case["iters"]
        return {"bytes": int(n * (18 * size + 16) + cells * 64), "flops": int(n * 750)}
    layers, rows = case["nhidden"], case.get("batch", 0)
    params = 256 * 32 + 256 * 256 * (layers - 1) + 4 * 256 + 257 * layers
    fwd = 2 * (256 * 32 + 256 * 256 * (layers - 1) + 4 * 256)
    if kind == "predict":
        rows = 2 * case["ni"] * case["nj"]
        return {"bytes": rows * (32 * 4 * 2 + 16) + params * 4, "flops": rows * (fwd + 12 * case["ni"])}
    steps = case.get("steps", 1)
    return {"bytes": steps * (rows * (32 * 2 + 16 + layers * 256 * 2 * 2) + params * 4 * (6 if kind == "train" else 1)),
            "flops": steps * rows * 3 * fwd}


# ---- the same in 64 bits, without the framework -------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _faces(x, y, tri):
    """Neighbour across face k (opposite node k) of every cell, -1 far field, -2 wall; the face's outward
    vector, its midpoint minus the cell's centroid, the cell's area."""
    n = len(tri)
    t = tri - 1
    p, q = t[:, [1, 2, 0]], t[:, [2, 0, 1]]
    key = (np.minimum(p, q).astype(np.int64) * len(x) + np.maximum(p, q)).ravel()
    o = np.argsort(key, kind="stable")
    ks = key[o]
    pair = np.flatnonzero(ks[1:] == ks[:-1])
    nb = np.full(3 * n, -1, np.int64)
    nb[o[pair]], nb[o[pair + 1]] = o[pair + 1] // 3, o[pair] // 3
    nb = nb.reshape(n, 3)
    mx, my = 0.5 * (x[p] + x[q]), 0.5 * (y[p] + y[q])
    nb[(nb < 0) & (np.abs(mx) < WALL_BOX) & (np.abs(my) < WALL_BOX)] = -2
    s = np.stack([y[q] - y[p], x[p] - x[q]], -1)
    cx, cy = x[t].mean(1), y[t].mean(1)
    r = np.stack([mx - cx[:, None], my - cy[:, None]], -1)
    area = 0.5 * np.abs((x[t[:, 1]] - x[t[:, 0]]) * (y[t[:, 2]] - y[t[:, 0]])
                        - (x[t[:, 2]] - x[t[:, 0]]) * (y[t[:, 1]] - y[t[:, 0]]))
    return nb, s, r, area


class _Flow:
    """The scheme in FP64 torch over the concatenated cells of one or more cases."""

    def __init__(self, case, parts):
        dev = _dev()
        self.case, off, cols = case, 0, []
        self.off = [0]
        for x, y, tri, ma, alpha in parts:
            nb, s, r, area = _faces(x, y, tri)
            n = len(tri)
            a = alpha * math.pi / 180.0
            fs = np.broadcast_to([math.cos(a), math.sin(a), 1.0 / (GAMMA * ma * ma)], (n, 3))
            cols.append((np.where(nb >= 0, nb + off, nb), s, r, area, fs))
            off += n
            self.off.append(off)
        nb, s, r, area, fs = [torch.from_numpy(np.concatenate([c[k] for c in cols])).to(dev) for k in range(5)]
        self.nb, self.s, self.r, self.area, self.fs = nb, s, r, area, fs
        self.inner = nb >= 0
        self.idx = torch.where(self.inner, nb, torch.arange(off, device=dev)[:, None])
        self.len = s.norm(dim=-1)
        self.n = s / self.len[..., None]
        self.bnd = (~self.inner).nonzero()
        self.wall = nb[self.bnd[:, 0], self.bnd[:, 1]] == -2
        self.clog = self.inner.sum(1).to(torch.float64)
        self.phi, self.frozen = None, False

    @staticmethod
    def prim(w):
        rho = w[..., 0]
        u, v = w[..., 1] / rho, w[..., 2] / rho
        p = (GAMMA - 1.0) * (w[..., 3] - 0.5 * rho * (u * u + v * v))
        return rho, u, v, p

    def ghosts(self, w):
        """Neighbour states [n, 3, 4] with the far-field and slip-wall ghosts filled in."""
        g = w[self.idx]
        c, k = self.bnd[:, 0], self.bnd[:, 1]
        wi, nx, ny = w[c], self.n[c, k, 0], self.n[c, k, 1]
        rho, u, v, p = self.prim(wi)
        a = torch.sqrt(GAMMA * p / rho)
        un = u * nx + v * ny
        wu, wv = u - 2 * un * nx, v - 2 * un * ny
        ui, vi, pa = self.fs[c, 0], self.fs[c, 1], self.fs[c, 2]
        out = un > 0
        pin = 0.5 * (pa + p - rho * a * (nx * (ui - u) + ny * (vi - v)))
        pb = torch.where(out, pa, pin)
        rb = torch.where(out, rho + (pa - p) / (a * a), 1.0 + (pin - pa) / (a * a))
        ub = torch.where(out, u + nx * (p - pa) / (rho * a), ui - nx * (pa - pin) / (rho * a))
        vb = torch.where(out, v + ny * (p - pa) / (rho * a), vi - ny * (pa - pin) / (rho * a))
        far = torch.stack([rb, rb * ub, rb * vb, pb / (GAMMA - 1.0) + 0.5 * rb * (ub * ub + vb * vb)], -1)
        wal = torch.stack([rho, rho * wu, rho * wv, wi[:, 3]], -1)
        g[c, k] = torch.where(self.wall[:, None], wal, far)
        return g

    def stage(self, w):
        """Residual (sum of the face fluxes) and local time step of state w."""
        case = self.case
        g = self.ghosts(w)
        mean = 0.5 * (w[:, None] + g)
        grad = torch.einsum("nkq,nkd->nqd", mean, self.s) / self.area[:, None, None]
        rho, u, v, p = self.prim(mean)
        sr = (u * self.s[..., 0] + v * self.s[..., 1]).abs() + torch.sqrt(GAMMA * p / rho) * self.len
        dt = (self.area * case["cfl"] / sr.sum(1)).clamp(max=0.1)
        d = torch.einsum("nqd,nkd->nkq", grad, self.r)
        if self.frozen and self.phi is not None:
            phi = self.phi
        else:
            hi = torch.maximum(w, g.amax(1))[:, None]
            lo = torch.minimum(w, g.amin(1))[:, None]
            d1 = torch.where(d > 0, hi, lo) - w[:, None]
            safe = torch.where(d == 0, torch.ones_like(d), d)
            if case["limiter"] in (1, 3):
                e2 = (case["k"] ** 3 * self.area * self.area.sqrt())[:, None, None]
                f = (d1 * d1 + e2 + 2 * d * d1) / (d1 * d1 + 2 * d * d + d1 * d + e2)
            else:
                f = (d1 / safe).clamp(max=1.0)
            phi = torch.where(d == 0, torch.ones_like(d), f)
            if case["limiter"] >= 2:
                phi = torch.where(self.inner[..., None], phi, math.inf).amin(1, keepdim=True).expand_as(d)
            self.phi = phi
        own = torch.where(self.inner[..., None], w[:, None] + d * phi, w[:, None])
        flat = own.reshape(-1, 4)
        oth = torch.where(self.inner[..., None], flat[self.slot()], g)
        return (self.roe(own, oth) * self.len[..., None]).sum(1), dt

    def slot(self):
        """Index into [3 n] of the same face seen from the neighbour."""
        if not hasattr(self, "_slot"):
            back = self.nb[self.idx]
            me = torch.arange(len(self.nb), device=self.nb.device)[:, None, None]
            # two cells of a mesh share at most one face
            k = (back == me).to(torch.uint8).argmax(-1)
            self._slot = self.idx * 3 + k
        return self._slot

    def roe(self, a, b):
        nx, ny = self.n[..., 0], self.n[..., 1]
        r0, u0, v0, p0 = self.prim(a)
        r1, u1, v1, p1 = self.prim(b)
        h0, h1 = (a[..., 3] + p0) / r0, (b[..., 3] + p1) / r1
        m0, m1 = u0 * nx + v0 * ny, u1 * nx + v1 * ny
        sl, sr = r0.sqrt(), r1.sqrt()
        rb = sl * sr
        ub, vb, hb = [(q0 * sl + q1 * sr) / (sl + sr) for q0, q1 in ((u0, u1), (v0, v1), (h0, h1))]
        q = ub * ub + vb * vb
        c = torch.sqrt((GAMMA - 1.0) * (hb - 0.5 * q))
        vc = ub * nx + vb * ny

        def fix(z):
            return torch.where(z.abs() < 0.05, (z * z + 0.0025) / 0.1, z.abs())
        l0, l1, l2 = fix(vc - c), fix(vc), fix(vc + c)
        dp, dv = p1 - p0, m1 - m0
        f0 = l0 * (dp - rb * c * dv) / (2 * c * c)
        f1 = l1 * ((r1 - r0) - dp / (c * c))
        f2 = l2 * (dp + rb * c * dv) / (2 * c * c)
        du, dw = u1 - u0, v1 - v0
        diss = torch.stack([
            f0 + f1 + f2,
            f0 * (ub - c * nx) + f1 * ub + l1 * rb * (du - dv * nx) + f2 * (ub + c * nx),
            f0 * (vb - c * ny) + f1 * vb + l1 * rb * (dw - dv * ny) + f2 * (vb + c * ny),
            f0 * (hb - c * vc) + 0.5 * f1 * q + l1 * rb * (ub * du + vb * dw - dv * vc) + f2 * (hb + c * vc)], -1)
        fl = torch.stack([r0 * m0, u0 * r0 * m0 + nx * p0, v0 * r0 * m0 + ny * p0, r0 * m0 * h0], -1)
        fr = torch.stack([r1 * m1, u1 * r1 * m1 + nx * p1, v1 * r1 * m1 + ny * p1, r1 * m1 * h1], -1)
        return 0.5 * (fl + fr - diss)

    def iterate(self, w):
        case = self.case
        w0 = w
        for c in (RK5 if case["stages"] == 5 else RK4):
            res, dt = self.stage(w)
            if case["sweeps"]:
                src = res
                for _ in range(case["sweeps"]):
                    nbs = (src[self.idx] * self.inner[..., None]).sum(1)
                    src = (nbs * case["irs_eps"] + res) / (1.0 + case["irs_eps"] * self.clog)[:, None]
                res = torch.where(res.abs() > src.abs(), src, res)
            w = w0 - c * dt[:, None] * res / self.area[:, None]
        return w

    def forces(self, w):
        out = []
        p = self.prim(w)[3]
        c, k = self.bnd[self.wall, 0], self.bnd[self.wall, 1]
        f = (p[c] - self.fs[c, 2])[:, None] * self.s[c, k]
        for lo, hi in zip(self.off[:-1], self.off[1:]):
            fx, fy = f[(c >= lo) & (c < hi)].sum(0).tolist()
            ca, sa = self.fs[lo, 0].item(), self.fs[lo, 1].item()
            out.append([(-fx * sa + fy * ca) / 0.5, (fx * ca + fy * sa) / 0.5])
        return np.array(out)


def _frequencies(seed=3, sigma=1.0):
    """The Fourier features' frequencies: normal numbers of a 64-bit xorshift* generator."""
    mask = (1 << 64) - 1
    st = (seed * 0x9E3779B97F4A7C15 + 777) & mask
    u = []
    for _ in range(32):
        st ^= st >> 12
        st ^= (st << 25) & mask
        st ^= st >> 27
        u.append((((st * 0x2545F4914F6CDD1D) & mask) >> 11) / 9007199254740992.0)
    f = [sigma * math.sqrt(-2.0 * math.log(u[2 * k] + 1e-300)) * math.cos(2.0 * math.pi * u[2 * k + 1])
         for k in range(16)]
    return np.array(f).reshape(8, 2)


def _features(x, y, tri, mach, alpha):
    dev = _dev()
    nb, _, _, _ = _faces(x, y, tri)
    cx, cy = x[tri - 1].mean(1), y[tri - 1].mean(1)
    c, k = np.nonzero(nb == -2)
    p, q = tri[c, (k + 1) % 3] - 1, tri[c, (k + 2) % 3] - 1
    g = [torch.from_numpy(v).to(dev) for v in (x[p], y[p], x[q] - x[p], y[q] - y[p])]
    px, py = torch.from_numpy(cx).to(dev), torch.from_numpy(cy).to(dev)
    d = []
    for a, b in zip(px.split(20000), py.split(20000)):
        t = (((a[:, None] - g[0]) * g[2] + (b[:, None] - g[1]) * g[3]) / (g[2] ** 2 + g[3] ** 2)).clamp(0.0, 1.0)
        d.append(((a[:, None] - g[0] - t * g[2]) ** 2 + (b[:, None] - g[1] - t * g[3]) ** 2).amin(1).sqrt())
    al = alpha * math.pi / 180.0
    out = np.zeros((len(tri), 32))
    out[:, 0], out[:, 1], out[:, 2] = cx, cy, np.log(torch.cat(d).cpu().numpy() + 1e-3)
    out[:, 3], out[:, 4], out[:, 5] = mach, math.sin(al), math.cos(al)
    ph = 2.0 * math.pi * (np.stack([cx, cy], 1) @ _frequencies().T)
    out[:, 6:22:2], out[:, 7:22:2] = np.sin(ph), np.cos(ph)
    return out


def _network(nhidden, flat, x, t=None):
    """Prediction, or loss and gradient, of the network in FP64."""
    dev = _dev()
    ws, o = [], 0
    for layer in range(nhidden + 1):
        rows, cols = (4 if layer == nhidden else 256), (32 if layer == 0 else 256)
        for shape in ((rows, cols), (rows,)):
            m = math.prod(shape)
            ws.append(torch.from_numpy(flat[o:o + m].astype(np.float64)).reshape(shape).to(dev)
                      .requires_grad_(t is not None))
            o += m
    h = torch.from_numpy(np.asarray(x, np.float64)).to(dev)
    for layer in range(nhidden + 1):
        h = h @ ws[2 * layer].T + ws[2 * layer + 1]
        if layer < nhidden:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    if t is None:
        return h.cpu().numpy()
    loss = ((h - torch.from_numpy(t.astype(np.float64)).to(dev)) ** 2).mean()
    loss.backward()
    return float(loss.detach()), np.concatenate([w.grad.cpu().numpy().ravel() for w in ws])


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None  # which samples a step takes is the framework's own choice
    if kind == "gradient":
        loss, g = _network(case["nhidden"], _weights(case["nhidden"], seed), *_samples(case["batch"], seed))
        return {"loss": loss, "gradient": g}
    if kind == "predict":
        f = _features(*_mesh(case["ni"], case["nj"], seed), 0.62, 1.1)
        mean, std = _normalisation()
        y = _network(case["nhidden"], _weights(case["nhidden"], seed), (f - mean) / std)
        return {"features": f, "prediction": y}
    cells = 2 * case["ni"] * case["nj"] * case.get("ncase", 1) * (0.25 if case.get("uneven") else 1.0)
    if cells * case["iters"] * case["stages"] > 1.0e9:
        return None  # minutes
    if kind == "solve":
        x, y, tri = _mesh(case["ni"], case["nj"], seed)
        parts = [(x, y, tri, case["ma"], case["alpha"])]
        w = _state(x, y, tri, case["ma"], case["alpha"], seed)
    else:
        specs = _batch(case, seed)
        arrays = {q[:3]: _mesh(*q[:3]) for q in specs}
        parts = [(*arrays[q[:3]], q[3], q[4]) for q in specs]
        w = np.concatenate([_state(*arrays[q[:3]], q[3], q[4], seed + c) for c, q in enumerate(specs)])
    flow = _Flow(case, parts)
    w = torch.from_numpy(w).to(_dev())
    norm, resd = None, []
    if case.get("frozen"):
        w1 = flow.iterate(w)
        norm = ((w1 - w)[:, 0] ** 2).sum()
        flow.frozen = True
    for _ in range(case["iters"]):
        w1 = flow.iterate(w)
        d = ((w1 - w)[:, 0] ** 2).sum()
        norm = d if norm is None else norm
        resd.append(torch.sqrt((d + 1e-32) / norm).item())
        w = w1
    forces = flow.forces(w)
    w = w.cpu().numpy()
    if kind == "solve":
        return {"state": w, "resd": np.array(resd), "forces": forces[0]}
    return {"states": [w[a:b] for a, b in zip(flow.off[:-1], flow.off[1:])], "forces": forces}
