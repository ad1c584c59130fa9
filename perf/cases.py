"""Workloads for timing the solver through its public entry points.

Each case is one job as a user's program runs it: the host state goes in, the solver does the
work on the GPU, and the whole result comes back.

* ``march``     the loop of cube.f90:71-79, nsteps RK4 calls each followed by the norm of v_r;
                optionally with the analytic source term and the energy diagnostics;
* ``record``    a forward run over a 3-D sound speed that samples p at receivers every step;
* ``batch``     independent runs with uneven step counts in one context (a set of sources);
* ``gradient``  the misfit gradient with respect to the sound speed (checkpointed adjoint);
* ``rhs``       one COMPUTE_RHS call on host arrays.

The shells, sponges and step counts follow ``solar_b200.configs``: the uniform shell of the
6 x 32^3 check run, the stratified 6 x 128^3 one, the 6 x 64^3 source batches and the 6 x 96^3
misfit gradient.  ``exact`` computes the same results in 64 bits with plain torch operations
(the discretisation of the reference written out once more, and its gradient by autograd).
"""
import math

import numpy as np
import torch

from solar_b200.configs import RSUN, Config, Source, Sponge, cfl_dt, model_stratified, model_uniform, outer_sponge
from solar_b200.solver import Solver

FORCING_ANALYTIC = 1
# The forced runs start where the source's envelope is half way up (its centre is at 0.65).
START = 0.45
# The norm printed by the reference's loop is that of v_r (cube.f90:77), field 4.
V_R = 4


def listed():
    return [
        # the check run every user starts with: small, bound by latency and launches
        dict(name="march 32x32 fp64", kind="march", nx=32, nr=32, precision="fp64", nfields=5, medium="uniform",
             steps=100, forced=False),
        # a small single-precision run with gravity, on a face that is no multiple of 32
        dict(name="march 48x40 fp32 gravity", kind="march", nx=48, nr=40, precision="fp32", nfields=5, medium="gravity",
             steps=80, forced=False),
        # a forced run with its energy diagnostics, odd sizes
        dict(name="march 80x50 fp64 forced", kind="march", nx=80, nr=50, precision="fp64", nfields=5, medium="gravity",
             steps=60, forced=True),
        # the stratified production shell in both precisions
        dict(name="march 128x128 fp32", kind="march", nx=128, nr=128, precision="fp32", nfields=4, medium="stratified",
             steps=100, forced=False),
        dict(name="march 128x128 fp64", kind="march", nx=128, nr=128, precision="fp64", nfields=5, medium="stratified",
             steps=50, forced=False),
        # a larger shell whose radial extent differs from its faces'
        dict(name="march 192x120 fp32", kind="march", nx=192, nr=120, precision="fp32", nfields=4, medium="stratified",
             steps=80, forced=False),
        # forward modelling of seismograms over a 3-D sound speed
        dict(name="record 160x96 fp64", kind="record", nx=160, nr=96, precision="fp64", nfields=5, medium="stratified",
             steps=40, receivers=32),
        # a batch of sources, one run each, of uneven length
        dict(name="batch 12 of 64x64 fp32", kind="batch", nx=64, nr=64, precision="fp32", nfields=4, medium="stratified",
             runs=12, least=40, most=160),
        # one misfit gradient in each precision, and a small one with two checkpoint levels
        dict(name="gradient 96x96 fp64", kind="gradient", nx=96, nr=96, precision="fp64", nfields=5, medium="stratified",
             steps=40, every=20, inner=20, receivers=32, adjoint_state=False),
        dict(name="gradient 96x96 fp32", kind="gradient", nx=96, nr=96, precision="fp32", nfields=4, medium="stratified",
             steps=60, every=20, inner=20, receivers=32, adjoint_state=False),
        dict(name="gradient 48x33 fp32 nested", kind="gradient", nx=48, nr=33, precision="fp32", nfields=4,
             medium="stratified", steps=40, every=20, inner=5, receivers=12, adjoint_state=True),
        # the right-hand side alone, on host arrays, as a host program that keeps its own stepping calls it
        dict(name="rhs 64x64 fp64", kind="rhs", nx=64, nr=64, precision="fp64", nfields=5, medium="gravity"),
    ]


def draw(rng):
    kind = rng.choice(["march"] * 5 + ["record", "batch", "gradient", "gradient", "rhs"])
    precision = rng.choice(["fp64", "fp32"])
    top = {"march": 160, "record": 128, "batch": 64, "gradient": 96, "rhs": 96}[kind]
    nx = 16 * int(round(math.exp(rng.uniform(math.log(32), math.log(top))) / 16))
    nr = int(round(math.exp(rng.uniform(math.log(24), math.log(min(top, 120))))))
    medium = rng.choice(["uniform", "stratified", "stratified", "gravity"])
    nfields = 5 if medium == "gravity" or precision == "fp64" else 4
    case = dict(kind=kind, nx=nx, nr=nr, precision=precision, nfields=nfields, medium=medium)
    if kind == "march":
        case.update(steps=rng.randint(30, 60), forced=rng.random() < 0.25)
    elif kind == "record":
        case.update(steps=rng.randint(20, 40), receivers=rng.randint(5, 40))
    elif kind == "batch":
        case.update(runs=rng.randint(3, 10), least=rng.randint(20, 40), most=rng.randint(50, 100))
    elif kind == "gradient":
        every = rng.randint(5, 10)
        case.update(steps=rng.randint(12, 20), every=every, inner=rng.choice([every, 3]), receivers=rng.randint(5, 32),
                    adjoint_state=rng.random() < 0.5)
    return case


# ------------------------------------------------------------------ inputs
def _config(case):
    nx, nr, medium = case["nx"], case["nr"], case["medium"]
    model = model_uniform(nr) if medium == "uniform" else model_stratified(nr)
    if case.get("forced"):
        # a sound speed in cm/s, with which the source's period of 350 s is 0.35 in the shell's units
        model[:, 1] *= RSUN / 1000
    if medium == "gravity":
        # g0 = 0.4 r in units of c(1)^2 / R after SOLAR_DATA's normalisation
        model[:, 5] = 0.4 * model[:, 0] * model[0, 1] ** 2 / RSUN
    sponge = Sponge() if medium == "uniform" else outer_sponge(nr)
    return Config("case", nx, nr, model, cfl_dt(nx, model), 0, sponge, [Source((0.0, 0.0, 0.9), 0.05)])


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _axes(case):
    """Tangents of the face coordinate and the radius, on the device."""
    dev = _device()
    g = -math.pi / 4 + torch.arange(case["nx"], dtype=torch.float64, device=dev) * (math.pi / 2) / (case["nx"] - 1)
    r = torch.as_tensor(_config(case).model[:, 0].copy(), device=dev)
    return torch.tan(g), r


def _face(z, X, Y):
    """Unit vectors of one face's points, X along xi and Y along eta (metric.f90:95-158)."""
    one = torch.ones_like(X)
    v = torch.stack([(one, X, Y), (-X, one, Y), (-one, -X, Y), (X, -one, Y), (-Y, X, one), (Y, X, -one)][z], -1)
    return v / v.norm(dim=-1, keepdim=True)


def _pulses(case, rng, count, out):
    """Sum of `count` seeded Gaussian pulses in every stored field, written into out[6, 5, nr, n, n]."""
    t, r = _axes(case)
    X, Y = torch.broadcast_tensors(t[None, :], t[:, None])
    lo, hi = float(r[0]), float(r[-1])
    centre = rng.standard_normal((5, count, 3))
    centre *= (lo + (hi - lo) * rng.uniform(0.25, 0.85, (5, count, 1))) / np.linalg.norm(centre, axis=2, keepdims=True)
    width = rng.uniform(0.05, 0.25, (5, count))
    amp = rng.uniform(0.5, 1.0, (5, count)) * rng.choice([-1.0, 1.0], (5, count))
    scale = (0.2, 0.1, 0.1, 0.1, 1.0)  # rho, v_xi, v_eta, v_r, p
    for z in range(6):
        u = _face(z, X, Y)
        for m in range(5):
            f = torch.zeros((len(r),) + X.shape, dtype=torch.float64, device=t.device)
            if m or case["nfields"] == 5:
                for c, w, a in zip(centre[m], width[m], amp[m]):
                    # |r u - c|^2 = r^2 - 2 r (u . c) + |c|^2
                    d2 = (r * r + float(c @ c))[:, None, None] - 2 * r[:, None, None] * (u @ torch.as_tensor(c, device=t.device))
                    f += scale[m] * float(a) * torch.exp(-d2 / (2 * float(w) ** 2))
            out[z, m].copy_(f)


def _state_of(case, seed, out=None):
    """The initial state of `seed`: a pinned host tensor [6, 5, nr, n, n] (or written into `out`)."""
    if out is None:
        out = torch.empty((6, 5, case["nr"], case["nx"], case["nx"]), dtype=torch.float64, pin_memory=torch.cuda.is_available())
    _pulses(case, np.random.default_rng(seed), 3, out)
    return out


def _blobs(case, seed):
    """3-D c^2: the radial one times (1 + a few smooth anomalies), [6, nr, n, n] on the device."""
    rng = np.random.default_rng(seed + 1)
    t, r = _axes(case)
    X, Y = torch.broadcast_tensors(t[None, :], t[:, None])
    c = torch.as_tensor(_config(case).model[:, 1].copy(), device=t.device)
    c = (c / c[0])[None, :, None, None].repeat(6, 1, case["nx"], case["nx"])
    centre = rng.standard_normal((8, 3))
    centre *= (float(r[-1]) * rng.uniform(0.75, 0.97, (8, 1))) / np.linalg.norm(centre, axis=1, keepdims=True)
    for z in range(6):
        u = _face(z, X, Y)
        rel = torch.zeros_like(c[z])
        for b in centre:
            d2 = (r * r + float(b @ b))[:, None, None] - 2 * r[:, None, None] * (u @ torch.as_tensor(b, device=t.device))
            rel += 0.02 * torch.exp(-d2 / (2 * 0.1 ** 2))
        c[z] *= 1 + rel
    return c * c


def _receivers(case, seed):
    """Receiver rows (zone, i, j, k), away from the planes that the radial filter zeroes, and observed traces."""
    rng = np.random.default_rng(seed + 2)
    m, n, nr = case["receivers"], case["nx"], case["nr"]
    loc = np.stack([rng.integers(0, 6, m).astype(float), rng.uniform(0, n - 1, m), rng.uniform(0, n - 1, m),
                    rng.uniform(6, nr - 7, m)], 1)
    step = np.arange(case["steps"])[:, None]
    data = 0.2 * np.sin(0.1 * step * rng.uniform(0.5, 2, m) + rng.uniform(0, 6.28, m))
    return loc, data


def _run_steps(case, seed):
    return np.random.default_rng(seed + 3).integers(case["least"], case["most"] + 1, case["runs"])


def prepare(case, seed):
    kind, cfg = case["kind"], _config(case)
    s = dict(case=case, out=None)
    c2 = None
    if kind in ("record", "gradient"):
        c2 = _blobs(case, seed).cpu().numpy()
        loc, s["data"] = _receivers(case, seed)
    runs = case.get("runs", 1)
    s["solver"] = Solver(cfg, precision=case["precision"], nfields=case["nfields"], nruns=runs, c2_3d=c2)
    if case.get("forced"):
        s["solver"].set_forcing(FORCING_ANALYTIC, k_center=case["nr"] // 2)
    if kind in ("record", "gradient"):
        s["solver"].set_receivers(loc)
    # the host keeps its states in pinned memory, as a program that moves them every job does
    shape = (runs,) + s["solver"].state_shape
    q = torch.empty(shape, dtype=torch.float64, pin_memory=True)
    for r in range(runs):
        _state_of(case, seed + 1000 * r, q[r])
    s["q0"] = q.numpy()
    if kind in ("march", "record", "batch"):
        s["out64"] = torch.empty(shape, dtype=torch.float64, pin_memory=True)
        if case["precision"] == "fp32":
            s["out32"] = torch.empty(shape, dtype=torch.float32)
    if kind == "batch":
        s["steps"] = _run_steps(case, seed)
    if kind == "gradient":
        s["solver"].set_state(s["q0"][0])
    return s


# ------------------------------------------------------------------ one pass
def _result(s, values):
    """Arrays in the run's own precision: an FP32 run's host program keeps single-precision results."""
    if s["case"]["precision"] == "fp64":
        return values
    return {k: np.asarray(v, dtype=np.float32) for k, v in values.items()}


def _states(s):
    """Read back every run's state; an FP32 run's into the program's single-precision array."""
    for r in range(s["solver"].nruns):
        s["solver"].get_state(r, out=s["out64"][r].numpy())
    if s["case"]["precision"] == "fp64":
        return s["out64"]
    return s["out32"].copy_(s["out64"])


def run(s):
    case, g = s["case"], s["solver"]
    kind = case["kind"]
    if kind == "rhs":
        return _result(s, {"rhs": g.compute_rhs(s["q0"][0])})
    if kind == "gradient":  # starts from, and leaves, the state set once
        d = g.misfit_gradient(case["steps"], case["every"], s["data"], want_lambda=case["adjoint_state"],
                              inner_every=case["inner"])
        return _result(s, {k: np.asarray(d[k]) for k in ("misfit", "grad_c", "lambda0") if k in d})
    for r in range(g.nruns):
        g.set_state(s["q0"][r], r)
    if kind == "march":
        if case["forced"]:
            g.set_clock(START, 0)
        got = {"norms": g.rk4_norms(case["steps"], V_R)}
        if case["forced"]:
            d = g.diag()
            got.update(energy=np.array(d["energy"]), mass=np.array(d["mass"]), max_abs_p=np.array(d["max_abs_p"]))
    elif kind == "record":
        got = {"traces": g.record(case["steps"])}
    else:
        g.rk4_runs(s["steps"])
        got = {}
    return dict(_result(s, got), state=_states(s))


def work(case):
    """Bytes: the state in and out, and per step what the 2N-storage scheme keeps between its passes (stage 1 reads
    q and writes q, w; stages 2-4 read and write both; stage 5 reads both and writes q; the filter reads and writes q)."""
    pts, F = 6 * case["nx"] ** 2 * case["nr"], case["nfields"]
    w = 8 if case["precision"] == "fp64" else 4
    step, flops = 20 * F * w, 5 * (100 + 12 * F) + 40 * F
    io = 16 * F
    kind = case["kind"]
    if kind == "rhs":
        return dict(bytes=pts * (io + 2 * F * w), flops=pts * 110)
    if kind in ("march", "record"):
        n = case["steps"]
    elif kind == "batch":
        n = case["runs"] * (case["least"] + case["most"]) / 2
        io *= case["runs"]
    else:
        # forward, recomputation (and its divergences), reverse: the transposed stages keep the adjoint state and
        # register, read c^2 and the divergence and update the gradient
        n = case["steps"]
        nested = 1 if case["inner"] < case["every"] else 0
        io = 8
        step = (2 + nested) * step + 5 * w + (20 * F + 5 * (2 * w + 16))
        flops = (2 + nested) * flops + 1.5 * flops
    return dict(bytes=pts * (io + n * step), flops=pts * n * flops)


# ------------------------------------------------------------------ the same results in 64 bits
_DRP = (0.79926643, -0.18941314, 0.02651995)                       # header:40-46
_ONE_SIDED = ((-2.192280339, 4.748611401, -5.108851915, 4.461567104, -2.833498741, 1.128328861, -0.203876371),
              (-0.209337622, -1.084875676, 2.147776050, -1.388928322, 0.768949766, -0.28181465, 0.048230454),
              (0.049041958, -0.468840357, -0.474760914, 1.273274737, -0.518484526, 0.166138533, -0.026369431))
_ALPHA = (0.0, -4.801594388477952e-01, -1.404247195200064e+00, -2.016477077503357e+00, -1.056444269767207e+00)
_BETA = (1.028639988104959e-01, 7.408540575766301e-01, 7.426530946683799e-01, 4.694937902357905e-01, 1.881733382887932e-01)
_FILTER = (0.6875, 0.234375, -0.09375, 0.015625)                   # header:99-105
_FILTER_R = (0.753906, 0.2050775, -0.1171875, 0.043945, -0.0097655, 0.0009765)
# (sending face, its edge, reversed) for the S, N, W, E ghosts of each face (derivative.f90:55-133, 374-452)
_ROUTES = (((5, "N", 0), (4, "S", 0), (3, "E", 0), (1, "W", 0)), ((5, "E", 1), (4, "E", 0), (0, "E", 0), (2, "W", 0)),
           ((5, "S", 1), (4, "N", 1), (1, "E", 0), (3, "W", 0)), ((5, "W", 0), (4, "W", 1), (2, "E", 0), (0, "W", 0)),
           ((0, "N", 0), (2, "N", 1), (3, "N", 1), (1, "N", 0)), ((2, "S", 1), (0, "S", 0), (3, "S", 0), (1, "S", 1)))


def _taps(f, dim, weights, sign):
    """sum_m w[m] (f[+m] + sign f[-m]) over the points `half` away from both ends of dimension dim (m = 1 ..)."""
    half = len(weights)
    n = f.shape[dim] - 2 * half
    acc = 0
    for m, w in enumerate(weights, 1):
        acc = acc + w * (f.narrow(dim, half + m, n) + sign * f.narrow(dim, half - m, n))
    return acc


class _Shell:
    """The discretised shell in plain torch: fields are [6, nr, n, n] (face, k, j, i)."""

    def __init__(self, case, c2=None):
        cfg, dev = _config(case), _device()
        self.n, self.nr, self.dt, self.dev = cfg.nx, cfg.nr, cfg.dt, dev
        n, nr, M = cfg.nx, cfg.nr, cfg.model
        f64 = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=dev)  # noqa: E731
        g = -math.pi / 4 + np.arange(n) * (math.pi / 2) / (n - 1)
        self.dxi = dxi = g[1] - g[0]
        t = np.tan(g)
        # radial rows (ic_acoustic_wave.f90:73-108, metric.f90:48-67)
        r, rho0, g0 = M[:, 0], M[:, 2] / M[0, 2], M[:, 5] * RSUN / M[0, 1] ** 2
        chi = lambda f: self._radial(f64(f)[None, :, None, None]).flatten().cpu().numpy() * (nr - 1)  # noqa: E731
        drdchi = chi(r)
        col = lambda v: f64(v)[None, :, None, None]  # noqa: E731
        self.r, self.drdchi, self.rho0_1d = r, drdchi, rho0
        self.facr, self.invr, self.rho0, self.drho0, self.g0 = col((nr - 1) / drdchi), col(1 / r), col(rho0), col(chi(rho0) / drdchi), col(g0)
        self.c2 = col((M[:, 1] / M[0, 1]) ** 2) if c2 is None else c2
        sp, k = cfg.sponge, np.arange(1, nr + 1)
        up = nr - sp.length + 1
        ratio = lambda a: (a.astype(np.float32) / np.float32(sp.length)).astype(np.float64)  # noqa: E731  sponge.f90:41-43
        upper, lower = sp.upper & (k >= up), sp.lower & (k <= sp.length)
        self.sigma = col(np.where(upper, sp.amp * ratio(np.maximum(k - up, 0)) ** sp.exp,
                                  np.where(lower, sp.amp * ratio(np.maximum(sp.length - k, 0)) ** sp.exp, 0.0)))
        inner = np.ones(nr)
        inner[[0, -1]] = 0
        self.inner = col(inner)
        # metric of a face (metric.f90:73-85), X along i and Y along j
        X, Y = f64(t)[None, :].expand(n, n), f64(t)[:, None].expand(n, n)
        C, D, delta = torch.sqrt(1 + X * X), torch.sqrt(1 + Y * Y), 1 + X * X + Y * Y
        self.X, self.Y, self.C, self.D, self.delta = X, Y, C, D, delta
        # (v_xi, v_eta) -> (v_theta, v_phi) on faces 1-4, 5 and 6 (transform.f90:19-56)
        sd, f = torch.sqrt(delta), 1 / torch.sqrt(delta - 1)
        polar = (f * X / D, f * Y / C, -f * sd * Y / D, f * sd * X / C)
        self.conv = [(X * Y / (C * D), -torch.ones_like(X), sd / (C * D), torch.zeros_like(X))] * 4 + [polar, tuple(-a for a in polar)]
        # Lagrange weights from an edge's points to the ghost positions of layer m (interpolation.f90:22-52)
        self.lag = []
        for m in (1, 2, 3):
            at = np.arctan(t / math.tan(g[-1] + m * dxi))
            W = np.zeros((n, n))
            W[0, m] = W[n - 1, n - 1 - m] = 1
            for q in range(1, n - 1):
                u = np.arange(max(0, q - 4), min(n, q + 5))
                for a in u:
                    b = u[u != a]
                    W[q, a] = np.prod((at[q] - g[b]) / (g[a] - g[b]))
            self.lag.append(W)
        self.ghosts = [[self._ghost(f64, t, g, z, e) for e in range(4)] for z in range(6)]

    def _ghost(self, f64, t, g, face, e):
        """(source face, its edge, and per layer: position, interpolation matrix, rotation of theta and phi)."""
        src, edge, rev = _ROUTES[face][e]
        layers = []
        for m in (1, 2, 3):
            hi, lo = math.tan(g[-1] + m * self.dxi), math.tan(g[0] - m * self.dxi)
            one = np.ones_like(t)
            # receiver-frame components at the sender's edge index (transform.f90:142-274)
            if src <= 3 and edge in "EW":
                X = lo if edge == "E" else hi
                th, ph = 0 * one, np.sqrt(1 + X * X) * np.sqrt(1 + t * t) / np.sqrt(1 + X * X + t * t)
            elif src >= 4:
                Y = hi if src == 4 else lo
                th, ph = -one, t * Y / np.sqrt(1 + t * t + Y * Y)
            else:
                top = edge == "N"
                sg = 1.0 if top else -1.0
                if src in (0, 2):
                    V, turn = (lo if (src == 0) == top else hi), 1.0
                else:
                    V, turn = (hi if src == 1 else lo), -1.0
                s1, s2, c = np.sqrt(t * t + V * V), np.sqrt(1 + t * t + V * V), np.sqrt(1 + t * t)
                th, ph = sg * c * V / s1, turn * sg * c / s1 * t / s2
            W = self.lag[m - 1]
            if rev:  # the receiver reverses the strip
                W, th, ph = W[::-1], th[::-1], ph[::-1]
            at = m if edge in "SW" else self.n - 1 - m
            layers.append((at, f64(W.copy()), f64(th.copy()), f64(ph.copy())))
        return src, edge, layers

    @staticmethod
    def _line(f, edge, at):
        return f[..., at, :] if edge in "SN" else f[..., at]

    def _strip(self, face, e, scalar=None, vector=None):
        """The three ghost lines of one edge, nearest first: [nr, n] each."""
        src, edge, layers = self.ghosts[face][e]
        got = []
        for at, W, th, ph in layers:
            if scalar is not None:
                got.append(self._line(scalar[src], edge, at) @ W.T)
                continue
            a = [self._line(c, edge, at) for c in self.conv[src]]
            vx, ve = (self._line(v[src], edge, at) for v in vector)
            got.append(th * ((a[0] * vx + a[1] * ve) @ W.T) + ph * ((a[2] * vx + a[3] * ve) @ W.T))
        return got

    def _halo(self, f, dim, scalar=None, vector=None):
        """f with three ghost lines on either side along xi (dim 3) or eta (dim 2)."""
        lo, hi = (2, 3) if dim == 3 else (0, 1)
        both = []
        for z in range(6):
            a, b = self._strip(z, lo, scalar, vector), self._strip(z, hi, scalar, vector)
            both.append((torch.stack(a[::-1], dim - 1), torch.stack(b, dim - 1)))
        return torch.cat([torch.stack([p[0] for p in both]), f, torch.stack([p[1] for p in both])], dim)

    def _radial(self, f):
        """d/dchi times dchi: the centred rows and the one-sided ones at both ends (derivative.f90:656-754)."""
        mid = _taps(f, 1, _DRP, -1)
        low = [sum(w * f[:, m] for m, w in enumerate(row)) for row in _ONE_SIDED]
        top = [-sum(w * f[:, f.shape[1] - 1 - m] for m, w in enumerate(row)) for row in _ONE_SIDED]
        return torch.cat([torch.stack(low, 1), mid, torch.stack(top[::-1], 1)], 1)

    def rhs(self, q, c2=None, source=None):
        """COMPUTE_RHS: q is the list rho, v_xi, v_eta, v_r, p."""
        rho, vx, ve, vr, p = q
        d = lambda f, dim: _taps(f, dim, _DRP, -1) / self.dxi  # noqa: E731
        X, Y, C, D, invr, rho0 = self.X, self.Y, self.C, self.D, self.invr, self.rho0
        px, py = d(self._halo(p, 3, scalar=p), 3), d(self._halo(p, 2, scalar=p), 2)
        gx, ge, gr = invr * (D * px + X * Y / D * py), invr * (C * py + X * Y / C * px), self.facr * self._radial(p)
        dx, dy = d(self._halo(vx, 3, vector=(vx, ve)), 3), d(self._halo(ve, 2, vector=(vx, ve)), 2)
        scale = self.delta / (C * D)
        div = invr * (scale / C * dx + scale / D * dy - X / D * vx - Y / C * ve) + self.facr * self._radial(vr) + 2 * vr * invr
        out = [-rho0 * div - vr * self.drho0, -gx / rho0, -ge / rho0, -gr / rho0 - rho * self.g0 / rho0,
               -(self.c2 if c2 is None else c2) * rho0 * div + rho0 * self.g0 * vr]
        if source is not None:
            out[3] = out[3] + source
        return out

    def filter(self, q):
        """FILTER_EXP (filter.f90:9-48); rows outside the face enter the eta filter unfiltered."""
        got = []
        for f in q:
            x = _FILTER[0] * f + _taps(self._halo(f, 3, scalar=f), 3, _FILTER[1:], 1)
            y = _FILTER[0] * x + _taps(self._halo(x, 2, scalar=f), 2, _FILTER[1:], 1)
            r = _FILTER_R[0] * y[:, 5:-5] + _taps(y, 1, _FILTER_R[1:], 1)
            zero = torch.zeros_like(y[:, :5])
            got.append(torch.cat([zero, r, zero], 1))
        return got

    def step(self, q, c2=None, source=None):
        """RK4 (timestep.f90:61-82): five stages of rhs, radial boundary planes, sponge and update, then the filter."""
        w = [torch.zeros_like(f) for f in q]
        for a, b in zip(_ALPHA, _BETA):
            rate = [self.inner * f for f in self.rhs(q, c2, source)]
            for m in (0, 3, 4):
                rate[m] = rate[m] - self.sigma * q[m]
            w = [a * x + self.dt * y for x, y in zip(w, rate)]
            q = [x + b * y for x, y in zip(q, w)]
        return self.filter(q)

    def source_of(self, case, time):
        """The analytic source of compute_rhs_acoustic.f90:92-104 at one time, centred at plane nr / 2."""
        dev, dxi, dchi = self.dev, self.dxi, 1.0 / (self.nr - 1)
        xyz = torch.stack([_face(z, self.X, self.Y) for z in range(6)])
        theta, phi = torch.arccos(xyz[..., 2]), torch.atan2(xyz[..., 1], xyz[..., 0])
        phi[1:] = torch.where(phi[1:] < 0, phi[1:] + 2 * math.pi, phi[1:])  # only the first zone's runs from -pi/4
        flat = torch.exp(-((theta - math.pi / 2) / (20 * dxi)) ** 2 - (phi / (20 * dxi)) ** 2)
        r = torch.as_tensor(self.r.copy(), device=dev)
        depth = torch.exp(-((r - r[case["nr"] // 2]) / (20 * dchi)) ** 2)
        u = time * RSUN / float(_config(case).model[0, 1]) - 650.0
        return math.exp(-u * u / (2 * 200.0 ** 2)) * math.cos(4 * math.pi * u / 700) * depth[None, :, None, None] * flat[:, None]

    def diag(self, q):
        area = (self.C * self.D) ** 2 / self.delta ** 1.5 * self.dxi ** 2
        dv = area * torch.as_tensor(self.r ** 2 * self.drdchi / (self.nr - 1), device=self.dev)[None, :, None, None]
        energy = 0.5 * ((self.rho0 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) + q[4] ** 2 / (self.rho0 * self.c2)) * dv).sum()
        return dict(energy=energy.cpu(), mass=(q[0] * dv).sum().cpu(), max_abs_p=q[4].abs().max().cpu())


def _sample(p, loc):
    """Trilinear samples of p on the receivers' faces."""
    got = []
    for f, x, y, z in loc:
        n, nr = p.shape[-1], p.shape[1]
        i, j, k = min(int(x), n - 2), min(int(y), n - 2), min(int(z), nr - 2)
        wx, wy, wz = (torch.tensor([1 - v, v], dtype=p.dtype, device=p.device) for v in (x - i, y - j, z - k))
        got.append(torch.einsum("kji,k,j,i->", p[int(f), k:k + 2, j:j + 2, i:i + 2], wz, wy, wx))
    return torch.stack(got)


def exact(case, seed):
    kind, dev = case["kind"], _device()
    pts = 6 * case["nx"] ** 2 * case["nr"]

    def fields(offset=0):
        q = _state_of(case, seed + offset)
        q = [q[:, m].to(dev) for m in range(5)]
        if case["nfields"] == 4:
            q[0] = torch.zeros_like(q[0])
        return q

    def whole(q):
        q = [torch.zeros_like(q[0]) if m == 0 and case["nfields"] == 4 else f for m, f in enumerate(q)]
        return torch.stack(q, 1)

    c2 = _blobs(case, seed).to(dev) if kind in ("record", "gradient") else None
    shell = _Shell(case, c2)
    if kind != "gradient":
        with torch.no_grad():
            if kind == "rhs":
                return {"rhs": whole(shell.rhs(fields())).cpu()}
            if kind == "batch":
                got = []
                for r, steps in enumerate(_run_steps(case, seed)):
                    q = fields(1000 * r)
                    for _ in range(int(steps)):
                        q = shell.step(q)
                    got.append(whole(q).cpu())
                return {"state": torch.stack(got)}
            q, loc = fields(), (_receivers(case, seed)[0] if kind == "record" else None)
            along = []
            for k in range(case["steps"]):
                q = shell.step(q, source=shell.source_of(case, START + k * shell.dt) if case.get("forced") else None)
                along.append(torch.sqrt(q[3].square().sum() / (pts / 6) * 6) if loc is None else _sample(q[4], loc))
            got = {"norms" if loc is None else "traces": torch.stack(along).cpu(), "state": whole(q)[None].cpu()}
            if case.get("forced"):
                got.update(shell.diag(q))
            return got
    from torch.utils.checkpoint import checkpoint

    loc, data = _receivers(case, seed)
    c = torch.sqrt(c2).requires_grad_()
    q0 = [f.requires_grad_() for f in fields()]
    q, misfit = q0, 0.0
    for k in range(case["steps"]):
        q = list(checkpoint(lambda c, *q: tuple(shell.step(list(q), c * c)), c, *q, use_reentrant=False))
        misfit = misfit + 0.5 * (_sample(q[4], loc) - torch.as_tensor(data[k], device=dev)).square().sum()
    grad = torch.autograd.grad(misfit, [c] + q0, allow_unused=True)
    got = {"misfit": misfit.detach().cpu(), "grad_c": grad[0].cpu()}
    if case["adjoint_state"]:
        got["lambda0"] = whole([torch.zeros_like(f) if a is None else a for a, f in zip(grad[1:], q0)]).cpu()
    return got
