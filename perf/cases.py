"""Performance cases of the elastic engine and its learned preconditioner.

Each case is one call that a program on this framework makes through the
public entry points (`efwi.engine.Propagator`, `efwi.cnn`): `listed()` names
the standing ones, `draw()` gives more of the same ranges, `prepare()` makes
what the program holds before the call, `run()` is one pass, `work()` what the
pass cannot do without and `exact()` the same outputs in 64 bits from plain
torch.

The misfit is returned as float32, as `FWI_ops_3d.fwi_ops` returns it.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "efwi-3d_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from efwi import cnn  # noqa: E402
from efwi.engine import Grid, Propagator, Shot  # noqa: E402

C16 = 16


def _dev() -> torch.device:
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ------------------------------------------------------------------- cases
def listed():
    """Sizes are padded cells; spacing 10 m and 0.8 ms unless a case says
    otherwise.  `rec` is the side of the square receiver grid."""
    return [
        # the smallest modelling call: the non-cubic grid of the parity tests,
        # where a launch is a few microseconds
        dict(name="forward_small", kind="forward", nz=26, nx=30, ny=28, npml=6, nt=120, shots=1,
             rec=4),
        # line-search trial of a 64^3 model (84^3 padded, nt 500, 32 x 32
        # receivers): the misfit of one shot
        dict(name="misfit_84", kind="misfit", nz=84, nx=84, ny=84, npml=10, nt=500, shots=1,
             rec=32),
        # its gradient by the reference's adjoint
        dict(name="gradient_84", kind="gradient", nz=84, nx=84, ny=84, npml=10, nt=500, shots=1,
             rec=32),
        # observed data of a 128^3 survey (152^3 padded): a launch carries
        # four shots
        dict(name="forward_batch_152", kind="forward", nz=152, nx=152, ny=152, npml=12, nt=100,
             shots=4, rec=64),
        # the headline call, the reference gradient at 152^3: two shots on
        # two lanes
        dict(name="gradient_152", kind="gradient", nz=152, nx=152, ny=152, npml=12, nt=100,
             shots=2, rec=64),
        # a field survey's ragged grid with the windowed misfit: three
        # shots on two lanes
        dict(name="gradient_ragged", kind="gradient", nz=75, nx=109, ny=91, npml=8, nt=150,
             shots=3, rec=21, win=True),
        # the gradient that the inversion and autograd run on: the exact
        # adjoint of a 96^3 model (120^3 padded), checkpoints in 2 GiB
        dict(name="exact_120", kind="exact", nz=120, nx=120, ny=120, npml=12, nt=200, shots=1,
             rec=48, ck_gib=2.0),
        # marine-style acquisition: every shot on its own aperture window of
        # a 256 x 256 x 160 model, 12.5 m
        dict(name="windows_forward", kind="windows", nz=184, nx=280, ny=280, npml=12, nt=40,
             shots=8, rec=64, wmin=120, wmax=216, dx=12.5, dt=1e-3),
        # pseudo-Hessian diagonal, an input of the preconditioner: four shots
        # of a 64^3 training model (80^3 padded)
        dict(name="illumination_80", kind="illumination", nz=80, nx=80, ny=80, npml=8, nt=150,
             shots=4, rec=31),
        # the preconditioner inside an L-BFGS iteration on the 128^3 model
        dict(name="net_infer_128", kind="net", D=128, H=128, W=128, train=False),
        # one training pair: 64^3, forward, cosine loss and all gradients
        dict(name="net_train_64", kind="net", D=64, H=64, W=64, train=True),
        # one layer forward and backward on a ragged volume
        dict(name="layer_ragged", kind="layer", D=93, H=117, W=141, relu=True),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "misfit", "gradient", "gradient", "exact", "windows",
                       "illumination", "net", "layer"])
    if kind in ("net", "layer"):
        d, h, w = (_logint(rng, 20, 140) for _ in range(3))
        if kind == "net":
            return dict(kind="net", D=d, H=h, W=w, train=rng.random() < 0.5)
        return dict(kind="layer", D=d, H=h, W=w, relu=rng.random() < 0.7)
    if kind == "windows":
        npml = rng.randint(8, 12)
        nz, nx, ny = rng.randint(60, 184), rng.randint(150, 280), rng.randint(150, 280)
        wmin = rng.randint(60, 120)
        return dict(kind="windows", nz=nz, nx=nx, ny=ny, npml=npml, nt=rng.randint(20, 40),
                    shots=rng.randint(2, 8), rec=rng.randint(8, 64), wmin=wmin,
                    wmax=rng.randint(wmin, 146), dx=12.5, dt=1e-3)
    lo, hi = 26, 152
    if kind in ("exact", "illumination"):
        hi = 110
    base = _logint(rng, lo, hi)
    nz, nx, ny = (min(hi, max(lo, int(base * rng.uniform(0.75, 1.25)))) for _ in range(3))
    npml = rng.randint(5, min(12, (min(nz, nx, ny) - 6) // 3))
    shots = rng.randint(1, 4)
    # time steps: bounded so that no case costs more than the 152^3 gradient
    top = 250e6 if kind in ("exact", "illumination") else 600e6
    nt = max(40, min(500, int(top / (nz * nx * ny * shots))))
    side = max(2, min(nx, ny) - 2 * npml)
    case = dict(kind=kind, nz=nz, nx=nx, ny=ny, npml=npml, nt=min(nt, rng.randint(60, 500)),
                shots=shots, rec=rng.randint(2, min(side, 64)))
    if kind in ("gradient", "misfit"):
        case["win"] = rng.random() < 0.4
    if kind == "exact":
        case["ck_gib"] = round(rng.uniform(0.5, 4.0), 2)
    return case


# ------------------------------------------------------------------ inputs
def _model(case, gen, dev):
    """Layered vp with smooth interfaces and Gaussian anomalies (1800 to
    4000 m/s, +-8 % vp, +-10 % vs, rho = 310 vp^0.25), on the padded grid,
    as (lambda, mu, rho / 1e3) float32."""
    n = (case["nz"], case["nx"], case["ny"])
    rnd = lambda *s: torch.rand(*s, generator=gen, dtype=torch.float64)  # noqa: E731
    p = case["npml"]
    ax = []
    for m in n:  # replicate padding of the model into the C-PML
        ax.append(torch.arange(m, dtype=torch.float64, device=dev).clamp(p, m - 1 - p))
    vps = torch.sort(1800.0 + 2000.0 * rnd(5)).values.tolist()
    cuts = torch.sort(rnd(4)).values.tolist()
    z = (ax[0] - p) / max(n[0] - 2 * p - 1, 1)
    vz = torch.full_like(z, vps[0])
    for k in range(4):
        vz = vz + (vps[k + 1] - vps[k]) * torch.sigmoid((z - cuts[k]) * 24.0)
    vp = vz[:, None, None].expand(n).clone()
    vs = vp / 1.732
    for _ in range(6):
        c, sg = rnd(3).tolist(), float(0.05 + 0.07 * rnd(1))
        s = [1.0 if float(v) < 0.5 else -1.0 for v in rnd(2)]
        g = 1.0
        for k in range(3):
            e = torch.exp(-0.5 * ((ax[k] - c[k] * n[k]) / (sg * n[k])) ** 2)
            g = g * e.reshape([-1 if j == k else 1 for j in range(3)])
        vp = vp * (1.0 + 0.08 * s[0] * g)
        vs = vs * (1.0 + 0.10 * s[1] * g)
    vp = vp.clamp(1500.0, 4300.0)
    rho = 310.0 * vp ** 0.25 / 1e3
    mu = vs * vs * rho
    lam = (vp * vp - 2.0 * vs * vs) * rho
    return [t.float().contiguous() for t in (lam, mu, rho)]


def _ricker(f0, nt, dt):
    e = (np.pi * f0) ** 2
    t = np.arange(nt) * dt - 1.2 / f0
    return ((1.0 - 2.0 * e * t * t) * np.exp(-e * t * t)).astype(np.float32)


def _grid(case):
    dx, dt = case.get("dx", 10.0), case.get("dt", 8e-4)
    f0 = max(8.0, 3.0 / (case["nt"] * dt))  # the wavelet fits the time axis
    return Grid(case["nz"], case["nx"], case["ny"], case["npml"], case["nt"], dx, dx, dx, dt, f0)


def _inputs(case, seed):
    """Model, survey and field records of one elastic case.  The records are
    a direct arrival with moveout plus band-limited noise."""
    dev = _dev()
    gen = torch.Generator().manual_seed(int(seed))
    g = _grid(case)
    p, nt = g.npml, g.nt
    model = _model(case, gen, dev)
    rnd = lambda *s: torch.rand(*s, generator=gen)  # noqa: E731
    mx, my = g.nx - 2 * p, g.ny - 2 * p
    xs = p + (np.arange(case["rec"]) * (mx - 1)) // max(case["rec"] - 1, 1)
    ys = p + (np.arange(case["rec"]) * (my - 1)) // max(case["rec"] - 1, 1)
    X, Y = (a.ravel().astype(np.int32) for a in np.meshgrid(xs, ys, indexing="ij"))
    Z = np.full(X.size, p + 2, np.int32)
    shots, wins = [], []
    for k in range(case["shots"]):
        u = rnd(8).tolist()
        if case["kind"] == "windows":
            w = [case["wmin"] + int((case["wmax"] - case["wmin"]) * v) for v in u[:2]]
            x0, y0 = int((g.nx - w[0]) * u[2]), int((g.ny - w[1]) * u[3])
            wins.append((x0, y0, w[0], w[1]))
            src = (p + 4, x0 + w[0] // 2, y0 + w[1] // 2)
        else:
            src = (p + 3, p + 2 + int((mx - 4) * u[0]), p + 2 + int((my - 4) * u[1]))
        s = Shot(src=src, z_rec=Z, x_rec=X, y_rec=Y)
        if case.get("win"):
            t0 = (0.3 * nt * g.dt * rnd(X.size)).numpy().astype(np.float32)
            s.win_start = t0
            s.win_end = (t0 + np.float32(0.6 * nt * g.dt)).astype(np.float32)
            s.weights = (0.5 + rnd(X.size)).numpy().astype(np.float32)
            s.src_weight = 0.5 + u[4]
        shots.append(s)
    stf = np.stack([_ricker(g.f0 * (1.0 + 0.05 * k), nt, g.dt) for k in range(len(shots))])
    obs = None
    if case["kind"] in ("misfit", "gradient", "exact"):
        t = torch.arange(nt, dtype=torch.float64, device=dev) * g.dt
        parts = []
        dgen = torch.Generator(device=dev).manual_seed(int(seed) + 1)
        e = (math.pi * g.f0) ** 2
        for s in shots:
            off = g.dx * np.sqrt((X - s.src[1]) ** 2 + (Y - s.src[2]) ** 2 + 1.0)
            off = torch.from_numpy(off).to(dev)[:, None]
            tau = t[None] - 1.2 / g.f0 - off / 2200.0
            d = (1.0 - 2.0 * e * tau * tau) * torch.exp(-e * tau * tau)
            d = d * (g.dx / off).clamp(max=1.0)
            d = d[None] + 0.02 * _smooth_t(torch.randn(3, X.size, nt, generator=dgen, device=dev,
                                                       dtype=torch.float64))
            parts.append((0.2 * d).float().reshape(-1))
        obs = torch.cat(parts)
    return dict(grid=g, model=model, shots=shots, stf=stf, obs=obs, wins=wins)


def _smooth_t(x):
    k = torch.hann_window(11, periodic=False, dtype=x.dtype, device=x.device)
    return F.conv1d(x.reshape(-1, 1, x.shape[-1]), (k / k.norm())[None, None],
                    padding=5).reshape(x.shape)


def _feats(case, seed):
    """(gradient, model, log-illumination) features, each of order one."""
    dev = _dev()
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    shp = (case["D"], case["H"], case["W"])
    low = torch.randn((1, 4) + tuple(max(2, s // 6) for s in shp), generator=gen, device=dev)
    v = F.interpolate(low, size=shp, mode="trilinear", align_corners=False)[0]
    v = v + 0.1 * torch.randn(v.shape, generator=gen, device=dev)
    g = v[0] / v[0].abs().max()
    return torch.stack([g, v[1] / v[1].std(), 0.5 + 0.2 * v[2]]).contiguous(), v[3].contiguous()


def _layer(case, seed):
    """Activations after a ReLU, a layer's weights and the loss's gradient."""
    dev = _dev()
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    shp = (case["D"], case["H"], case["W"], C16)
    x = torch.randn(shp, generator=gen, device=dev).relu_().to(torch.bfloat16)
    w = torch.randn(27, C16, C16, generator=gen, device=dev) * math.sqrt(2.0 / (27 * C16))
    b = 0.1 * torch.randn(C16, generator=gen, device=dev)
    gy = torch.randn(shp, generator=gen, device=dev).to(torch.bfloat16)
    return x, w, b, gy


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        feats, target = _feats(case, seed)
        return dict(case=case, net=cnn.Preconditioner(seed=int(seed) % 1000).to(_dev()),
                    feats=feats, target=target)
    if kind == "layer":
        x, w, b, gy = _layer(case, seed)
        return dict(case=case, x=x.requires_grad_(True), w=w.requires_grad_(True),
                    b=b.requires_grad_(True), gy=gy)
    d = _inputs(case, seed)
    P = Propagator(d["grid"], if_win=bool(case.get("win")))
    if "ck_gib" in case:
        P.set_checkpoint_budget(int(case["ck_gib"] * (1 << 30)))
    P.set_survey(d["shots"], d["stf"])
    return dict(case=case, P=P, model=d["model"], obs=d["obs"], wins=d["wins"],
                ids=list(range(case["shots"])))


# --------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "net":
        net, feats = state["net"], state["feats"]
        if not case["train"]:
            with torch.no_grad():
                return net(feats)
        net.zero_grad(set_to_none=True)
        pred = net(feats)
        loss = _cosine(pred, state["target"])
        loss.backward()
        return {"pred": pred.detach(), "loss": loss.detach(),
                "grads": [p.grad for p in net.parameters()]}
    if kind == "layer":
        y = cnn.Conv3dBF16.apply(state["x"], state["w"], state["b"], case["relu"], False)
        dx, dw, db = torch.autograd.grad(y, (state["x"], state["w"], state["b"]), state["gy"])
        return {"y": y.detach(), "dx": dx, "dw": dw, "db": db}
    P, ids = state["P"], state["ids"]
    P.set_model(*state["model"])  # every evaluation brings a model
    if kind == "forward":
        return P.forward(ids)
    if kind == "misfit":
        return torch.tensor([P.misfit(ids, state["obs"])], dtype=torch.float32)
    if kind == "windows":
        return P.forward_windows(ids, state["wins"])
    if kind == "illumination":
        return list(P.illumination(ids))
    mode = "exact" if kind == "exact" else "reference"
    J, gl, gm, gr = P.gradient(ids, state["obs"], mode=mode)
    return {"misfit": torch.tensor([J], dtype=torch.float32), "lam": gl, "mu": gm, "rho": gr}


def _cosine(pred, target):
    p, t = pred.reshape(-1), target.reshape(-1)
    return 1.0 - torch.dot(p, t) / (torch.linalg.vector_norm(p) * torch.linalg.vector_norm(t))


# ------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass: per time step and shot 120 B a cell
    and 48 B a C-PML slab cell forward, three times that and the six model
    and image volumes for a gradient; a layer reads and writes its volume."""
    kind = case["kind"]
    if kind in ("net", "layer"):
        v = case["D"] * case["H"] * case["W"]
        layer = 2.0 * 27 * C16 * C16 * v
        if kind == "layer":
            return {"bytes": 32.0 * v * 5, "flops": 3 * layer}
        n = 4
        fwd = (3 * 4 + 32.0 * (2 * n - 1) + 4) * v
        return {"bytes": fwd * (3 if case["train"] else 1),
                "flops": n * layer * (3 if case["train"] else 1)}
    nz, p, nt = case["nz"], case["npml"], case["nt"]

    def step(nx, ny):
        n = nz * nx * ny
        s = 2 * p * (nx * ny + nz * ny + nz * nx)
        return n, 120.0 * n + 48.0 * s

    if kind == "windows":
        m = (case["wmin"] + case["wmax"]) / 2
        n, b = step(m, m)
    else:
        n, b = step(case["nx"], case["ny"])
    steps = (nt - 1.0) * case["shots"]
    flops = 160.0 * n
    if kind in ("gradient", "exact"):
        b, flops = 3.0 * b + 24.0 * n, 3 * flops
    elif kind == "illumination":
        b, flops = 2.0 * b + 24.0 * n, 2 * flops
    return {"bytes": b * steps, "flops": flops * steps}


# -------------------------------------------------- the same in 64 bits
_C1, _C2 = 9.0 / 8.0, 1.0 / 24.0
_AX = {"z": 0, "x": 1, "y": 2}
# memory variables: (differentiated field, axis, half point, update stage)
_PSI_S = [("vz", "z", 0), ("vx", "z", 1), ("vy", "z", 1), ("vx", "x", 0), ("vz", "x", 1),
          ("vy", "x", 1), ("vy", "y", 0), ("vz", "y", 1), ("vx", "y", 1)]
_PSI_V = [("szz", "z", 1), ("sxz", "z", 0), ("syz", "z", 0), ("sxx", "x", 1), ("sxz", "x", 0),
          ("sxy", "x", 0), ("syy", "y", 1), ("syz", "y", 0), ("sxy", "y", 0)]
_FIELDS = ["vz", "vx", "vy", "szz", "sxx", "syy", "sxz", "sxy", "syz"]


def _profile(n, p, dh, f0, dt):
    """C-PML rows 1/K, a, b at integer and at half points."""
    amax, L = 2.0 * math.pi * (f0 / 2.0), p * dh
    d0 = -(8.0 + 1.0) * 3000.0 * math.log(0.0008) / (2.0 * L)
    rows = np.zeros((2, 3, n))
    for half in (0, 1):
        for i in range(n):
            d, K, al = 0.0, 1.0, 0.0
            h = 0.5 * half
            for depth in ((p - i - h) * dh, (p - n + i + h) * dh):
                if depth >= 0.0:
                    x = depth / L
                    d, K = d0 * (0.25 * x + 0.75 * x ** 8), 1.0 + x ** 8
                    al = max(amax * (1.0 - x), 0.0)
            b = math.exp(-(d / K + al) * dt)
            a = d * (b - 1.0) / (K * (d + K * al)) if abs(d) > 1e-6 else 0.0
            rows[half, :, i] = 1.0 / K, a, b
    return rows


class _Exact:
    """The scheme on one grid in float64: the forward half-steps, the
    reference's reverse sweep, and (through autograd) the exact adjoint."""

    def __init__(self, grid, model, src, rec, stf, dev):
        f32 = lambda v: float(np.float32(v))  # noqa: E731
        self.g, self.dev = grid, dev
        self.n = (grid.nz, grid.nx, grid.ny)
        self.dt = f32(grid.dt)
        self.h = (f32(grid.dz), f32(grid.dx), f32(grid.dy))
        self.lam, self.mu, rho = (m.to(dev, torch.float64) for m in model)
        self.set_rho(rho)
        self.src, self.rec = src, rec
        self.stf = self._taper(stf)
        p = grid.npml
        self.cf, self.slab_s, self.slab_v = [], [], []
        for k, m in enumerate(self.n):
            r = torch.from_numpy(_profile(m, p, self.h[k], f32(grid.f0), self.dt))[:, :, 2:-2]
            view = [-1 if j == k else 1 for j in range(3)]
            self.cf.append([[r[q, c].reshape(view).to(dev) for c in range(3)] for q in (0, 1)])
            i = torch.arange(m, device=dev)[2:-2]
            self.slab_s.append(((i < p) | (i > m - p - 1)).double().reshape(view))
            self.slab_v.append(((i < p) | (i > m - p)).double().reshape(view))
        self.slab_v[0] = self.slab_s[0]

    def set_rho(self, rho):
        self.rho = rho
        self.buoy = self.c(1.0 / rho)

    def _taper(self, stf):
        nt, dt = self.g.nt, self.dt
        t3, off = nt * dt, nt * dt * 0.001
        out = stf.astype(np.float64).copy()
        for it in range(nt):
            t = it * dt
            w = 1.0
            if t < off:
                w = math.sin(math.pi / 2 * t / off)
            elif t >= t3 - off:
                w = math.cos(math.pi / 2 * (t - t3 + off) / off) if t < t3 else 0.0
            out[it] *= w * w
        return out

    # interior views and differences
    @staticmethod
    def s(f, ax, k):
        ix = [slice(2, -2)] * 3
        n = f.shape[ax]
        ix[ax] = slice(2 + k, n - 2 + k)
        return f[tuple(ix)]

    def c(self, f):
        return self.s(f, 0, 0)

    def dm(self, f, ax):
        return (_C1 * (self.s(f, ax, 0) - self.s(f, ax, -1)) -
                _C2 * (self.s(f, ax, 1) - self.s(f, ax, -2))) / self.h[ax]

    def dp(self, f, ax):
        return (_C1 * (self.s(f, ax, 1) - self.s(f, ax, 0)) -
                _C2 * (self.s(f, ax, 2) - self.s(f, ax, -1))) / self.h[ax]

    def dq(self, f, ax):  # the velocity update's difference of sxy along x
        return (_C1 * (self.s(f, ax, 0) - self.s(f, ax, -1)) -
                _C2 * (self.s(f, ax, -1) - self.s(f, ax, -2))) / self.h[ax]

    def zeros(self):
        z = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        st = {f: z for f in _FIELDS}
        m = self.c(z)
        st.update({("m",) + k: m for k in _PSI_S + _PSI_V})
        return st

    def _stage(self, st, keys, slab, store=True):
        """C-PML-modified derivatives of one stage; new memory variables."""
        d, mem = {}, {}
        for f, a, half in keys:
            ax = _AX[a]
            v = self.dp(st[f], ax) if half else self.dm(st[f], ax)
            if f == "sxy" and a == "x":
                v = self.dq(st[f], ax)
            ki, ca, cb = self.cf[ax][half]
            m = slab[ax] * (cb * st[("m", f, a, half)] + ca * v)
            mem[("m", f, a, half)] = m
            d[f, a] = torch.where(slab[ax] > 0, v * ki + m, v)
        return d, mem

    def stress(self, st, it):
        d, mem = self._stage(st, _PSI_S, self.slab_s)
        l, u, dt = self.c(self.lam), self.c(self.mu), self.dt
        e = {"z": d["vz", "z"], "x": d["vx", "x"], "y": d["vy", "y"]}
        div = l * (e["z"] + e["x"] + e["y"])
        add = {"szz": div + 2 * u * e["z"], "sxx": div + 2 * u * e["x"],
               "syy": div + 2 * u * e["y"], "sxz": u * (d["vx", "z"] + d["vz", "x"]),
               "sxy": u * (d["vx", "y"] + d["vy", "x"]), "syz": u * (d["vy", "z"] + d["vz", "y"])}
        out = dict(st)
        out.update(mem)
        amp = 2250000.0 * self.stf[it] * self.dt
        for f, v in add.items():
            new = st[f] + F.pad(v * dt, (2,) * 6)
            if f in ("szz", "sxx", "syy"):
                b = torch.zeros_like(new)
                b[tuple(self.src)] = amp
                new = new + b
            out[f] = new
        return out

    def velocity(self, st):
        d, mem = self._stage(st, _PSI_V, self.slab_v)
        bt = self.buoy * self.dt
        out = dict(st)
        out.update(mem)
        out["vz"] = st["vz"] + F.pad((d["szz", "z"] + d["sxz", "x"] + d["syz", "y"]) * bt, (2,) * 6)
        out["vx"] = st["vx"] + F.pad((d["sxz", "z"] + d["sxx", "x"] + d["sxy", "y"]) * bt, (2,) * 6)
        out["vy"] = st["vy"] + F.pad((d["syz", "z"] + d["sxy", "x"] + d["syy", "y"]) * bt, (2,) * 6)
        return out

    def sample(self, st):
        z, x, y = self.rec
        return torch.stack([st[f][z, x, y] for f in ("vx", "vy", "vz")])

    def forward(self, shell=None):
        """Traces [3][nrec][nt]; with `shell` (cell indices) also the state
        at the shell cells before every step."""
        st, tr, saved = self.zeros(), [], []
        tr.append(self.sample(st))
        for it in range(self.g.nt - 1):
            if shell is not None:
                saved.append(torch.stack([st[f].reshape(-1)[shell] for f in _FIELDS]))
            st = self.velocity(self.stress(st, it))
            tr.append(self.sample(st))
        self.state = st
        return torch.stack(tr, 2), saved

    def window(self, shot, if_win):
        """Time taper of the misfit, [nrec][nt] (or [1][nt]); its times are
        float32 seconds, so that a sample falls on the same side of an edge."""
        nt, dt, f4 = self.g.nt, np.float32(self.g.dt), np.float32
        t = np.arange(nt, dtype=f4) * dt
        tmax = f4(nt) * dt
        if if_win:
            t0 = np.clip(shot.win_start.astype(f4), 0, tmax)[:, None]
            t3 = np.clip(shot.win_end.astype(f4), 0, tmax)[:, None]
            wt = shot.weights.astype(np.float64)[:, None] * float(f4(shot.src_weight))
        else:
            t0, t3, wt = np.zeros((1, 1), f4), np.full((1, 1), tmax, f4), 1.0
        off = (t3 - t0) * f4(0.005)
        t1, t2 = t0 + off, t3 - off
        up = np.sin(np.pi / 2 * (t - t0).astype(np.float64) / (t1 - t0))
        down = np.cos(np.pi / 2 * (t - t2).astype(np.float64) / (t3 - t2))
        w = np.where((t >= t0) & (t < t1), up, 0.0)
        w = np.where((t >= t1) & (t < t2), 1.0, w)
        w = np.where((t >= t2) & (t < t3), down, w)
        return torch.from_numpy(w * w * wt).to(self.dev)

    def residual(self, tr, obs, w):
        r = w * (obs.double() - tr)
        keep = torch.ones_like(r)
        keep[:, :, 0] = 0.0
        return r * keep

    # ---- the reference's gradient
    def shell_cells(self):
        p, lo = self.g.npml, self.g.npml - 2
        box, inner = [], []
        for k, n in enumerate(self.n):
            hi = n - p + 1
            i = torch.arange(n, device=self.dev)
            view = [-1 if j == k else 1 for j in range(3)]
            box.append(((i >= max(lo, 2)) & (i <= min(hi, n - 3))).reshape(view))
            inner.append(((i > lo + 4) & (i < hi - 4)).reshape(view))
        m = (box[0] & box[1] & box[2]) & ~(inner[0] & inner[1] & inner[2])
        return m.reshape(-1).nonzero()[:, 0]

    def reference_gradient(self, obs, w):
        g, dt, cell = self.g, self.dt, self.shell_cells()
        tr, saved = self.forward(cell)
        res = self.residual(tr, obs, w)
        J = (res * res).sum()
        res = res * w
        p, c, b = g.npml, self.c, self.buoy
        l, u = c(self.lam), c(self.mu)
        l2u = l + 2 * u
        inr = torch.ones((), device=self.dev, dtype=torch.bool)
        for k, n in enumerate(self.n):
            i = torch.arange(n, device=self.dev)[2:-2]
            inr = inr & ((i >= p) & (i <= n - 1 - p)).reshape([-1 if j == k else 1 for j in range(3)])
        f = {k: self.state[k] for k in _FIELDS}
        z0 = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        a = {k: z0.clone() for k in _FIELDS}
        ps = {(ax, q): z0.clone() for ax in "zxy" for q in ("A", "B1", "B2", "S", "T1", "T2")}
        gl, gm, gr = (torch.zeros_like(b) for _ in range(3))
        sl = {k: self.slab_s[_AX[k]] for k in "zxy"}
        K, A, B, Kh, Ah, Bh = ({k: self.cf[_AX[k]][q][r] for k in "zxy"}
                               for q, r in ((0, 0), (0, 1), (0, 2), (1, 0), (1, 1), (1, 2)))
        dm = lambda v, ax: -self.dm(v, _AX[ax])  # noqa: E731
        dp = lambda v, ax: -self.dp(v, _AX[ax])  # noqa: E731
        vshell, sshell = ("vz", "vx", "vy"), ("szz", "sxx", "syy", "sxz", "sxy", "syz")

        def put(d, k, v, where):
            d[k] = F.pad(torch.where(where, v, c(d[k])), (2,) * 6)

        def restore(names, it):
            for n in names:
                t = f[n].reshape(-1).clone()
                t[cell] = saved[it][_FIELDS.index(n)]
                f[n] = t.reshape(self.n)

        def mem(ax, q, coef, add):
            m = c(ps[ax, q])
            ps[ax, q] = F.pad(torch.where(sl[ax] > 0, coef[ax] * m + add * dt, m), (2,) * 6)

        def adj_velocity(it):
            nax = c(a["vx"]) + (l2u * dp(a["sxx"], "x") * K["x"] + l * dp(a["szz"], "x") * K["x"] +
                                l * dp(a["syy"], "x") * K["x"] + u * Kh["z"] * dm(a["sxz"], "z") +
                                u * Kh["y"] * dm(a["sxy"], "y")) * dt
            nax = nax + sl["x"] * A["x"] * dp(ps["x", "A"], "x") + \
                sl["z"] * Ah["z"] * dm(ps["z", "B1"], "z") + sl["y"] * Ah["y"] * dm(ps["y", "B2"], "y")
            naz = c(a["vz"]) + (l2u * dp(a["szz"], "z") * K["z"] + l * dp(a["sxx"], "z") * K["z"] +
                                l * dp(a["syy"], "z") * K["z"] + u * Kh["y"] * dm(a["syz"], "y") +
                                u * Kh["x"] * dm(a["sxz"], "x")) * dt
            naz = naz + sl["z"] * A["z"] * dp(ps["z", "A"], "z") + \
                sl["y"] * Ah["y"] * dm(ps["y", "B1"], "y") + sl["x"] * Ah["x"] * dm(ps["x", "B1"], "x")
            nay = c(a["vy"]) + (l2u * dp(a["syy"], "y") * K["y"] + l * dp(a["sxx"], "y") * K["y"] +
                                l * dp(a["szz"], "y") * K["y"] + u * Kh["x"] * dm(a["sxy"], "x") +
                                u * Kh["z"] * dm(a["syz"], "z")) * dt
            nay = nay + sl["y"] * A["y"] * dp(ps["y", "A"], "y") + \
                sl["x"] * Ah["x"] * dm(ps["x", "B2"], "x") + sl["z"] * Ah["z"] * dm(ps["z", "B2"], "z")
            mem("x", "S", Bh, b * nax), mem("z", "T1", B, b * nax), mem("y", "T2", B, b * nax)
            mem("x", "T1", B, b * naz), mem("z", "S", Bh, b * naz), mem("y", "T1", B, b * naz)
            mem("x", "T2", B, b * nay), mem("z", "T2", Bh, b * nay), mem("y", "S", B, b * nay)
            z, x, y = self.rec
            for n, v, k in (("vx", nax, 0), ("vy", nay, 1), ("vz", naz, 2)):
                t = F.pad(v, (2,) * 6)
                t.index_put_((z, x, y), res[k, :, it], accumulate=True)
                a[n] = t

        def adj_stress():
            bt = b * dt
            sxz = c(a["sxz"]) + dp(a["vz"], "x") * K["x"] * bt + dp(a["vx"], "z") * K["z"] * bt + \
                sl["x"] * A["x"] * dp(ps["x", "T1"], "x") + sl["z"] * A["z"] * dp(ps["z", "T1"], "z")
            sxy = c(a["sxy"]) + dp(a["vy"], "x") * K["x"] * bt + dp(a["vx"], "y") * K["y"] * bt + \
                sl["x"] * A["x"] * dp(ps["x", "T2"], "x") + sl["y"] * A["y"] * dp(ps["y", "T2"], "y")
            syz = c(a["syz"]) + dp(a["vz"], "y") * K["y"] * bt + dp(a["vy"], "z") * K["z"] * bt + \
                sl["y"] * A["y"] * dp(ps["y", "T1"], "y") + sl["z"] * A["z"] * dp(ps["z", "T2"], "z")
            sxx = c(a["sxx"]) + bt * dm(a["vx"], "x") * Kh["x"] + sl["x"] * Ah["x"] * dm(ps["x", "S"], "x")
            szz = c(a["szz"]) + bt * dm(a["vz"], "z") * Kh["z"] + sl["z"] * Ah["z"] * dm(ps["z", "S"], "z")
            syy = c(a["syy"]) + bt * dm(a["vy"], "y") * Kh["y"] + sl["y"] * Ah["y"] * dm(ps["y", "S"], "y")
            mem("x", "B1", Bh, sxz * u), mem("z", "B1", Bh, sxz * u)
            mem("y", "B2", Bh, sxy * u), mem("x", "B2", Bh, sxy * u)
            mem("y", "B1", Bh, syz * u), mem("z", "B2", Bh, syz * u)
            mem("x", "A", B, l * szz + l2u * sxx + l * syy)
            mem("z", "A", B, l2u * szz + l * sxx + l * syy)
            mem("y", "A", B, l * szz + l * sxx + l2u * syy)
            for n, v in (("sxz", sxz), ("sxy", sxy), ("syz", syz), ("sxx", sxx), ("szz", szz),
                         ("syy", syy)):
                a[n] = F.pad(v, (2,) * 6)

        nt = g.nt
        adj_velocity(nt - 1)
        adj_stress()
        for it in range(nt - 2, -1, -1):
            dz = self.dp(f["szz"], 0) + self.dm(f["sxz"], 1) + self.dm(f["syz"], 2)
            dx = self.dm(f["sxz"], 0) + self.dp(f["sxx"], 1) + self.dm(f["sxy"], 2)
            dy = self.dm(f["syz"], 0) + self.dq(f["sxy"], 1) + self.dp(f["syy"], 2)
            gr += torch.where(inr, (c(a["vz"]) * dz + c(a["vx"]) * dx + c(a["vy"]) * dy) * dt * b * b, 0.0)
            for n, d in (("vz", dz), ("vx", dx), ("vy", dy)):
                put(f, n, c(f[n]) - d * b * dt, inr)
            if it > 0:
                adj_velocity(it)
            restore(vshell, it)
            amp = 2250000.0 * self.stf[it] * dt
            for n in ("szz", "sxx", "syy"):
                f[n] = f[n].clone()
                f[n][tuple(self.src)] -= amp
            ez, ex, ey = self.dm(f["vz"], 0), self.dm(f["vx"], 1), self.dm(f["vy"], 2)
            exz = self.dp(f["vx"], 0) + self.dp(f["vz"], 1)
            exy = self.dp(f["vx"], 2) + self.dp(f["vy"], 1)
            eyz = self.dp(f["vy"], 0) + self.dp(f["vz"], 2)
            div = ez + ex + ey
            az, axx, ay = c(a["szz"]), c(a["sxx"]), c(a["syy"])
            gl -= torch.where(inr, (az + axx + ay) * div * dt, 0.0)
            gm -= torch.where(inr, (2 * (az * ez + axx * ex + ay * ey) + c(a["sxz"]) * exz +
                                    c(a["syz"]) * eyz + c(a["sxy"]) * exy) * dt, 0.0)
            for n, e in (("szz", l * div + 2 * u * ez), ("sxx", l * div + 2 * u * ex),
                         ("syy", l * div + 2 * u * ey), ("sxz", u * exz), ("sxy", u * exy),
                         ("syz", u * eyz)):
                put(f, n, c(f[n]) - e * dt, inr)
            if it > 0:
                adj_stress()
            restore(sshell, it)
        return J, [F.pad(v, (2,) * 6) for v in (gl, gm, gr)]

    # ---- the exact gradient
    def exact_gradient(self, obs, w, seg=8):
        par = [t.clone().requires_grad_(True) for t in (self.lam, self.mu, self.rho)]
        st = self.zeros()
        keys, nt = list(st), self.g.nt
        tr0 = self.sample(st)[:, :, None]

        def segment(lo, hi, lam, mu, rho, *vals):
            self.lam, self.mu = lam, mu
            self.set_rho(rho)
            s, out = dict(zip(keys, vals)), []
            for it in range(lo, hi):
                s = self.velocity(self.stress(s, it))
                out.append(self.sample(s))
            return (torch.stack(out, 2),) + tuple(s[k] for k in keys)

        vals, parts = [st[k] for k in keys], [tr0]
        for lo in range(0, nt - 1, seg):
            r = checkpoint(segment, lo, min(lo + seg, nt - 1), *par, *vals, use_reentrant=False)
            parts.append(r[0])
            vals = list(r[1:])
        res = self.residual(torch.cat(parts, 2), obs, w)
        J = (res * res).sum()
        return J.detach(), list(torch.autograd.grad(J, par))

    # ---- the pseudo-Hessian diagonal
    def illumination(self):
        st, dt2, nt = self.zeros(), self.dt ** 2, self.g.nt
        hl, hm, hb = (torch.zeros_like(self.buoy) for _ in range(3))
        for it in range(nt - 1):
            mid = self.stress(st, it)
            d, _ = self._stage(mid, _PSI_V, self.slab_v)
            st = self.velocity(mid)
            hb += dt2 * ((d["szz", "z"] + d["sxz", "x"] + d["syz", "y"]) ** 2 +
                         (d["sxz", "z"] + d["sxx", "x"] + d["sxy", "y"]) ** 2 +
                         (d["syz", "z"] + d["sxy", "x"] + d["syy", "y"]) ** 2)
            if it + 1 <= nt - 2:
                e, _ = self._stage(st, _PSI_S, self.slab_s)
                n = [e["vz", "z"], e["vx", "x"], e["vy", "y"]]
                hl += 3 * dt2 * (n[0] + n[1] + n[2]) ** 2
                hm += dt2 * (4 * (n[0] ** 2 + n[1] ** 2 + n[2] ** 2) +
                             (e["vx", "z"] + e["vz", "x"]) ** 2 + (e["vx", "y"] + e["vy", "x"]) ** 2 +
                             (e["vy", "z"] + e["vz", "y"]) ** 2)
        return [F.pad(v, (2,) * 6) for v in (hl, hm, hb * self.buoy ** 4)]


def _exact_elastic(case, seed):
    dev, d = _dev(), _inputs(case, seed)
    g, kind = d["grid"], case["kind"]
    nrec = len(d["shots"][0].z_rec)
    nt, traces, J, img, off = g.nt, [], 0.0, None, 0
    for k, s in enumerate(d["shots"]):
        model, rec = d["model"], (s.z_rec, s.x_rec, s.y_rec)
        src, gg = s.src, g
        keep = np.ones(nrec, bool)
        if kind == "windows":
            x0, y0, wx, wy = d["wins"][k]
            keep = (s.x_rec >= x0) & (s.x_rec < x0 + wx) & (s.y_rec >= y0) & (s.y_rec < y0 + wy)
            rec = (s.z_rec[keep], s.x_rec[keep] - x0, s.y_rec[keep] - y0)
            model = [m[:, x0:x0 + wx, y0:y0 + wy] for m in model]
            src = (s.src[0], s.src[1] - x0, s.src[2] - y0)
            gg = Grid(g.nz, wx, wy, g.npml, nt, g.dz, g.dx, g.dy, g.dt, g.f0)
        rec = [torch.from_numpy(np.ascontiguousarray(r)).long().to(dev) for r in rec]
        E = _Exact(gg, model, src, rec, d["stf"][k], dev)
        if kind in ("forward", "windows"):
            tr = torch.zeros(3, nrec, nt, dtype=torch.float64, device=dev)
            tr[:, torch.from_numpy(keep).to(dev)] = E.forward()[0]
            traces.append(tr.reshape(-1))
            continue
        if kind == "illumination":
            out = E.illumination()
        else:
            obs = d["obs"][off:off + 3 * nrec * nt].reshape(3, nrec, nt)
            off += obs.numel()
            w = E.window(s, bool(case.get("win")))
            if kind == "misfit":
                r = E.residual(E.forward()[0], obs, w)
                J, out = J + float((r * r).sum()), []
            else:
                j, out = (E.exact_gradient if kind == "exact" else E.reference_gradient)(obs, w)
                J += float(j)
        img = out if img is None else [a + b for a, b in zip(img, out)]
    if traces:
        return torch.cat(traces)
    if kind == "illumination":
        return img
    J = torch.tensor([J], dtype=torch.float64)
    if kind == "misfit":
        return J
    return {"misfit": J, "lam": img[0], "mu": img[1], "rho": img[2]}


def _conv64(x, w, b):
    """x [16, D, H, W], w [27, co, ci] in float64: one product per tap."""
    D, H, W = x.shape[1:]
    xp = F.pad(x, (1,) * 6)
    y = b.reshape(-1, 1, 1, 1) if b is not None else 0.0
    for t in range(27):
        i, j, k = t // 9, (t // 3) % 3, t % 3
        v = xp[:, i:i + D, j:j + H, k:k + W].reshape(x.shape[0], -1)
        y = y + (w[t] @ v).reshape(-1, D, H, W)
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        x, w, b, gy = _layer(case, seed)
        X = x.double().permute(3, 0, 1, 2).contiguous().requires_grad_(True)
        W = w.to(torch.bfloat16).double().requires_grad_(True)
        B = b.double().requires_grad_(True)
        y = _conv64(X, W, B)
        y = y.relu() if case["relu"] else y
        dx, dw, db = torch.autograd.grad(y, (X, W, B), gy.double().permute(3, 0, 1, 2))
        return {"y": y.detach().permute(1, 2, 3, 0), "dx": dx.permute(1, 2, 3, 0), "dw": dw, "db": db}
    if kind == "net":
        feats, target = _feats(case, seed)
        net = cnn.Preconditioner(seed=int(seed) % 1000).to(_dev())  # its seeded weights
        W = [p.detach().to(torch.bfloat16).double().requires_grad_(True) for p in net.w]
        B = [p.detach().double().requires_grad_(True) for p in net.b]
        h = F.pad(feats.to(torch.bfloat16).double(), (0,) * 6 + (0, C16 - feats.shape[0]))
        for k in range(len(W)):
            h = _conv64(h, W[k], B[k])
            if k + 1 < len(W):
                h = h.relu()
        if not case["train"]:
            return h[0].detach()
        loss = _cosine(h[0], target.double())
        grads = torch.autograd.grad(loss, W + B)
        return {"pred": h[0].detach(), "loss": loss.detach(), "grads": list(grads)}
    return _exact_elastic(case, seed)
