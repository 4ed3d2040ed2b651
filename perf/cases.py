"""Performance cases of the phase-space solver, its adjoint and its splines.

Every case is work that a program using this package has it do, through the
public classes:

kind "run"      VlasovSolver21Spline: `steps` steps with the statistics row
                every `every` steps, as run() does, and the grid read back
                into page-locked memory at the end, as before a snapshot
kind "adjoint"  adjoint_forward / adjoint_backward of `steps` steps with a
                checkpoint every `every`: gradients with respect to the
                initial grid and the delayed-kernel chain values
kind "theta"    final_density as a torch.autograd function of the profile's
                parameters: the final radial density and its gradient
kind "spline"   LocalSpline2: assign and build a batch of slices, evaluate it
                at a set of points

A grid is given by vertices along r and v_r and cells along J (Pres + 1,
Ures[0] + 1 and Ures[1] of the options).  Grids of FP32 handles are returned
as float32 (their storage type), everything else as float64.  exact() is the
same mathematics in plain 64-bit torch, without the package.
"""
import math
import random

import numpy as np
import torch

from vlasolve_b200 import VlasovSolver21Spline
from vlasolve_b200.adjoint import DensityProblem, final_density
from vlasolve_b200.spline import LocalSpline2

# r range, |v_r| range, J range and J scale of each profile's grid, time step
PROFILES = {
    "UDF": ((0.01, 25.0), 2.0, (0.0, 1.6), "quadratic", 0.005),
    "Plummer": ((0.01, 25.0), 3.0, (0.0, 2.0), "quadratic", 0.005),
    "Hernquist": ((0.01, 50.0), 3.0, (0.0, 3.0), "quadratic", 0.0025),
    "PLDF": ((0.01, 200.0), 1.5, (0.0, 1.6), "quadratic", 0.005),
    # the Hernquist profile's default ranges (J logarithmic)
    "HernquistDefault": ((0.01, 250.0), 1.45, (1.0e-4, 12.96), "logarithmic", 0.025),
}
STATS = ("Mass", "E", "Ek", "Ep", "S", "L1", "L2")
MOST_CELLS, MOST_WORK = 513 * 513 * 256, 513 * 513 * 256 * 200


def listed():
    def case(name, kind, profile, nr, nu, nj, precision, steps, every, **kw):
        return dict(name=name, kind=kind, profile=profile, nr=nr, nu=nu, nj=nj,
                    precision=precision, steps=steps, every=every, **kw)

    return [
        # one step of a test-sized grid looked at after every step: the
        # interactive and unit-test use, where launches and latency count
        case("step_udf_33x33x8_fp64", "run", "UDF", 33, 33, 8, "fp64", 1, 1),
        # a small survey run: the Hernquist default grid with the unlinked
        # step and a delayed kernel wider than its first cell
        case("run_hernquist_91x81x80_fp64_nolink", "run", "HernquistDefault", 91, 81, 80, "fp64",
             50, 25, noLinking=True, kernelBufferSize=2),
        # the reference's default UDF grid in FP64, its default statsEvery
        case("run_udf_201x201x200_fp64", "run", "UDF", 201, 201, 200, "fp64", 50, 25),
        # the production grid of isotropic models in the production precision
        case("run_plummer_257x257x128_fp32", "run", "Plummer", 257, 257, 128, "fp32", 100, 25),
        # ragged lines (no power of two, no 16-byte rows), linked FP32
        case("run_udf_395x307x77_fp32", "run", "UDF", 395, 307, 77, "fp32", 100, 25),
        # the benchmark workload: 67.4 M cells, FP32 storage
        case("run_hernquist_513x513x256_fp32", "run", "Hernquist", 513, 513, 256, "fp32", 200,
             25),
        # the same lines in FP64, half the slices: the accuracy runs
        case("run_hernquist_513x513x128_fp64", "run", "Hernquist", 513, 513, 128, "fp64", 100,
             25),
        # the longest lines in use (1025 vertices), an eighth of the slices
        case("run_pldf_1025x1025x64_fp32", "run", "PLDF", 1025, 1025, 64, "fp32", 50, 25),
        # gradient of a density loss with respect to the whole initial state
        case("adjoint_udf_257x257x128_fp64", "adjoint", "UDF", 257, 257, 128, "fp64", 50, 10),
        # the same in FP32 storage on a grid whose adjoint field exceeds L2
        case("adjoint_hernquist_513x513x64_fp32", "adjoint", "Hernquist", 513, 513, 64, "fp32",
             20, 10),
        # a fit of profile parameters: density and gradient in one pass
        case("theta_udf_129x129x64_fp64", "theta", "UDF", 129, 129, 64, "fp64", 40, 10),
        # the spline level used by itself: a batch of slices, a point set
        dict(name="spline_16x513x513_fp64", kind="spline", nr=513, nu=513, nj=16,
             precision="fp64", points=1000000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "adjoint", "theta", "spline"])
    precision = rng.choice(["fp64", "fp32"])
    if kind == "spline":
        nr, nu = _log(rng, 33, 1025), _log(rng, 33, 1025)
        nj = max(1, min(_log(rng, 1, 64), 16 * 513 * 513 // (nr * nu)))
        return dict(kind=kind, nr=nr, nu=nu, nj=nj, precision=precision,
                    points=_log(rng, 1000, 1000000))
    if kind == "run":
        profile = rng.choice(sorted(PROFILES))
        nr, nu, nj = _log(rng, 33, 1025), _log(rng, 33, 1025), _log(rng, 8, 256)
        nj = max(8, min(nj, MOST_CELLS // 2 // (nr * nu)))
        every = rng.choice([1, 5, 25])
        steps = every * rng.randint(1, max(1, 100 // every))
        return dict(kind=kind, profile=profile, nr=nr, nu=nu, nj=nj, precision=precision,
                    steps=steps, every=every, noLinking=rng.random() < 0.2,
                    kernelBufferSize=rng.choice([0, 0, 1, 3]))
    top = 513 if kind == "adjoint" else 161
    profile = rng.choice(["UDF", "Plummer", "Hernquist"]) if kind == "adjoint" else "UDF"
    nr, nu, nj = _log(rng, 49, top), _log(rng, 49, top), _log(rng, 8, 64)
    every = rng.randint(3, 10)
    return dict(kind=kind, profile=profile, nr=nr, nu=nu, nj=nj,
                precision=precision if kind == "adjoint" else "fp64",
                steps=every * rng.randint(1, 3), every=every)


# ------------------------------------------------------------------ inputs
def _options(case, seed):
    """The grid.*, solver.* and init.* options of a case; the profile's
    parameters come from the seed."""
    (r0, r1), um, (j0, j1), js, dt = PROFILES[case["profile"]]
    init = case["profile"].replace("Default", "")
    rng = random.Random(seed)
    o = dict(type=init, Pmin=r0, Pmax=r1, Pres=case["nr"] - 1, Pscale="logarithmic",
             Umin=(-um, j0), Umax=(um, j1), Ures=(case["nu"] - 1, case["nj"]),
             Uscale=("linear", js), dt=dt, M=1.0)
    if init == "UDF":
        o.update(R0=rng.uniform(1.8, 2.2), alpha=rng.uniform(0.45, 0.55), smoothingRadius=0.5)
    elif init == "PLDF":
        o.update(n=rng.uniform(0.95, 1.05), alpha=rng.uniform(0.9, 1.1), eta=0.1,
                 smoothingRadius=0.5)
    else:
        o.update(R0=rng.uniform(0.9, 1.1))
    if case.get("noLinking"):
        o["noLinking"] = 1
    if case.get("kernelBufferSize"):
        o["kernelBufferSize"] = case["kernelBufferSize"]
    return o


def _dbins(case, seed):
    """A cotangent of the radial bins, smooth as a density residual's is."""
    g = np.random.default_rng(seed)
    x = np.linspace(0.0, 1.0, case["nr"])
    return sum(a * np.sin((k + 1) * np.pi * x + p)
               for k, (a, p) in enumerate(g.uniform(-1.0, 1.0, (6, 2))))


def _spline_inputs(case, seed):
    g = np.random.default_rng(seed)
    x = np.linspace(0, 1, case["nr"])[None, None, :]
    y = np.linspace(-1, 1, case["nu"])[None, :, None]
    a = g.uniform(0.5, 1.5, (3, case["nj"], 1, 1))
    data = a[0] * np.exp(-6 * a[1] * (y * y + x)) + 0.1 * np.cos(9 * a[2] * x * y)
    n = case["points"]
    xx = np.exp(g.uniform(math.log(0.01001), math.log(24.99), n))
    yy = g.uniform(-1.999, 1.999, n)
    return data, xx, yy, g.integers(0, case["nj"], n)


def prepare(case, seed):
    if case["kind"] == "spline":
        data, xx, yy, sl = _spline_inputs(case, seed)
        sp = LocalSpline2((0.01, -2.0), (25.0, 2.0), (case["nr"] - 1, case["nu"] - 1),
                          scale=("logarithmic", "linear"), nslices=case["nj"],
                          precision=case["precision"])
        return dict(kind="spline", spline=sp, data=data, xx=xx, yy=yy, slices=sl,
                    single=case["precision"] != "fp64")
    opt = _options(case, seed)
    if case["kind"] == "theta":
        p = DensityProblem(opt, precision=case["precision"], nsteps=case["steps"],
                           checkpoint_every=case["every"])
        theta = torch.tensor([opt["R0"], opt["alpha"], opt["smoothingRadius"]],
                             dtype=torch.float64, requires_grad=True)
        return dict(kind="theta", problem=p, theta=theta,
                    weight=torch.from_numpy(_dbins(case, seed)[:-1].copy()))
    s = VlasovSolver21Spline(opt, precision=case["precision"])
    state = dict(kind=case["kind"], solver=s, steps=case["steps"], every=case["every"],
                 single=case["precision"] != "fp64")
    if case["kind"] == "adjoint":
        state["dbins"] = _dbins(case, seed)
        return state
    grid = torch.empty(s.shape, dtype=torch.float64, pin_memory=True)
    state["grid"], state["view"] = grid, grid.numpy()
    state["grid32"] = torch.empty(s.shape, dtype=torch.float32) if state["single"] else None
    return state


# -------------------------------------------------------------------- work
def run(state):
    kind = state["kind"]
    if kind == "run":
        s = state["solver"]
        rows = []
        for _ in range(state["steps"] // state["every"]):
            s.step(state["every"])
            row = s.stats()
            rows.append([row[k] for k in STATS])
        s.get_f_into(state["view"])
        if state["single"]:
            return dict(f=state["grid32"].copy_(state["grid"]),
                        stats=torch.tensor(rows, dtype=torch.float32))
        return dict(f=state["view"], stats=np.array(rows))
    if kind == "adjoint":
        s = state["solver"]
        s.adjoint_forward(state["steps"], state["every"])
        bins = s.moments()[0]
        df0, dchain = s.adjoint_backward(state["dbins"])
        if state["single"]:
            return tuple(torch.from_numpy(x).float() for x in (bins, df0, dchain))
        return bins, df0, dchain
    if kind == "theta":
        theta = state["theta"]
        rho = final_density(theta, state["problem"])
        grad, = torch.autograd.grad((rho * state["weight"]).sum(), theta)
        return rho.detach(), grad
    sp = state["spline"]
    sp.assign(state["data"])
    sp.build()
    v = sp.evaluate(state["xx"], state["yy"], state["slices"])
    return v.astype(np.float32) if state["single"] else v


def work(case):
    """One step reads and writes the grid once in each of its two sub-steps
    (the kick needs the whole grid's mass); per cell and step three spline
    solves, a four-tap and a sixteen-tap gather."""
    cells = case["nr"] * case["nu"] * case["nj"]
    es = 8 if case["precision"] == "fp64" else 4
    if case["kind"] == "spline":
        return {"bytes": cells * (8 + 2 * es) + case["points"] * 32,
                "flops": cells * 16 + case["points"] * 60}
    drifts = case["steps"] * (2 if case.get("noLinking") else 1)
    b, f = drifts * cells * 4 * es, drifts * cells * 75
    if case["kind"] == "run":
        b += case["steps"] // case["every"] * cells * es + cells * 8
    else:  # forward, recomputation, transposed step in FP64
        b, f = 2 * b + case["steps"] * cells * 32, 4 * f
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact
def _t(x):
    return torch.as_tensor(x, dtype=torch.float64, device="cuda")


def _scale(a, b, n, kind, vertex=True):
    lin = lambda p, q: p + (q - p) / n * np.arange(n + 1)  # noqa: E731
    s = (lin(a, b) if kind == "linear" else np.exp(lin(math.log(a), math.log(b)))
         if kind == "logarithmic" else lin(math.sqrt(a), math.sqrt(b)) ** 2)
    if vertex:
        s[0], s[-1] = a, b
        return s
    return 0.5 * (s[:-1] + s[1:])


def _solve_matrix(n):
    """(n + 2) x n: node values to natural cubic B-spline coefficients."""
    a = torch.zeros(n + 2, n + 2, dtype=torch.float64, device="cuda")
    k = torch.arange(1, n + 1, device="cuda")
    a[k, k - 1], a[k, k], a[k, k + 1] = 1 / 6, 4 / 6, 1 / 6
    a[0, :3] = a[-1, -3:] = _t([1.0, -2.0, 1.0])
    return torch.linalg.inv(a)[:, 1:-1].contiguous()


def _weights(t):
    s = 1 - t
    return (s ** 3 / 6, (1 + 3 * s + 3 * s * s - 3 * s ** 3) / 6,
            (1 + 3 * t + 3 * t * t - 3 * t ** 3) / 6, t ** 3 / 6)


def _drift(R, U, J, dt):
    """(r, v_r) a time dt back along the free orbit of angular momentum J,
    through the pericentre where the orbit passes it."""
    h2 = U * U + J * J / (R * R)
    out = U > 0
    peri = torch.sqrt(torch.clamp(R * R * h2 - J * J, min=0.0)) / h2
    turn = out & (peri < dt)
    q = (R * U).abs()
    q = torch.where(turn, (q - h2 * peri).abs(), q)
    rt = torch.sqrt(q * q + J * J) / torch.sqrt(h2)
    h2 = torch.where(turn, J * J / (rt * rt), h2)
    q = torch.where(turn, torch.zeros_like(q), q)
    sgn = torch.where(out & ~turn, 1.0, -1.0)
    left = torch.where(turn, dt - peri, torch.full_like(q, dt))
    r = torch.sqrt((q - sgn * h2 * left) ** 2 + J * J) / torch.sqrt(h2)
    return r, sgn * torch.sqrt(torch.clamp(h2 - J * J / (r * r), min=0.0))


def _taps(C, j, i, x, k, y):
    """Values of the splines C [j][row][column] at (row k + y, column i + x)."""
    pitch, flat = C.shape[2], C.reshape(-1)
    at = (j * C.shape[1] + k) * pitch + i
    wx, wy = _weights(x), _weights(y)
    v = 0
    for a in range(4):
        v = v + wy[a] * sum(wx[b] * flat[at + (a * pitch + b)] for b in range(4))
    return v


class _Model:
    """The solver's step in 64-bit torch on one grid."""

    def __init__(self, o):
        nr, nu, nj = o["Pres"] + 1, o["Ures"][0] + 1, o["Ures"][1]
        self.o, self.shape, self.dt = o, (nj, nu, nr), o["dt"]
        R = _scale(o["Pmin"], o["Pmax"], nr - 1, o["Pscale"])
        U = _scale(o["Umin"][0], o["Umax"][0], nu - 1, "linear")
        J = _scale(o["Umin"][1], o["Umax"][1], nj, o["Uscale"][1], False)
        JV = _scale(o["Umin"][1], o["Umax"][1], nj, o["Uscale"][1])
        dJ = np.where(np.arange(nj) >= nu - 1, 0.0, np.diff(JV))
        self.R, self.U, self.J = _t(R), _t(U), _t(J)
        self.dR, self.dU = _t(np.append(np.diff(R), 0.0)), _t(np.append(np.diff(U), 0.0))
        self.ct = _t(8 * math.pi ** 2 * J * dJ)
        self.bu = self.dU + torch.cat([_t([0.0]), self.dU[:-1]])
        self.coef = self.dt / self.R ** 2
        self.Pr, self.Pu = _solve_matrix(nr), _solve_matrix(nu)
        self.hu = (nu - 1) / (U[-1] - U[0])
        self.hr = (nr - 1) / (math.log(R[-1]) - math.log(R[0]))
        self.kr = R[o.get("kernelBufferSize", 0)]
        self.dth = 0.5 * self.dt if o.get("noLinking") else self.dt
        grid = torch.meshgrid(self.J, self.U, self.R, indexing="ij")
        r, u = _drift(grid[2], grid[1], grid[0], self.dth)
        inner = r < self.kr
        out = (r >= R[-1]) | (r <= R[0]) | (u >= U[-1]) | (u <= U[0])
        self.gather = torch.nonzero((~inner & ~out).reshape(-1)).reshape(-1)
        self.foot = self._place(r.reshape(-1)[self.gather], u.reshape(-1)[self.gather],
                                self.gather // (nr * nu))
        # delayed-kernel chains: positions at every dth until the orbit is
        # back outside the kernel; the last one is read from the spline
        self.cell = torch.nonzero(inner.reshape(-1)).reshape(-1)
        c = [g.reshape(-1)[self.cell] for g in grid[::-1]]
        self.n = torch.zeros_like(self.cell)
        seen, t, live = [], self.dth, torch.ones_like(self.cell, dtype=torch.bool)
        while self.cell.numel() and bool(live.any()):
            r, u = _drift(*c, t)
            self.n += live.long()
            seen.append((r, u))
            live = live & (r < self.kr)
            t += self.dth
        self.first = torch.cumsum(self.n, 0) - self.n
        n = int(self.n.sum())
        self.er, self.eu, self.ej = (torch.zeros(n, dtype=torch.float64, device="cuda")
                                     for _ in range(3))
        self.tail = torch.zeros(n, dtype=torch.bool, device="cuda")
        for e, (r, u) in enumerate(seen):
            m = self.n > e
            at = self.first[m] + e
            self.er[at], self.eu[at], self.ej[at] = r[m], u[m], c[2][m]
        if n:
            last = self.first + self.n - 1
            self.tail[last] = True
            tr, tu = self.er[last], self.eu[last]
            ok = (tu > U[0]) & (tu < U[-1])
            self.tail_ok = ok
            self.tail_foot = self._place(tr[ok], tu[ok], (self.cell // (nr * nu))[ok])

    def _place(self, r, u, j):
        x = (torch.log(r) - math.log(float(self.R[0]))) * self.hr
        y = (u - self.U[0]) * self.hu
        i, k = torch.trunc(x), torch.trunc(y)
        return j, i.long(), x - i, k.long(), y - k

    def profile(self, r, u, j, th=None):
        o = dict(self.o, **(th or {}))
        t = o["type"]
        l2 = (j / r) ** 2
        if t == "UDF":
            s2 = o["alpha"] / (5 * o["R0"])
            f = (0.5 * (1 + torch.erf((o["R0"] - r) / o["smoothingRadius"]))
                 * (3 / (4 * math.pi * o["R0"] ** 3)) * (2 * math.pi * s2) ** -1.5
                 * torch.exp(-(u * u + l2) / (2 * s2)))
            return torch.clamp(f, min=1e-200)
        if t == "PLDF":
            n, R0 = o["n"], 1 / o["eta"]
            so = (3 - n) / (5 - 2 * n) * o["eta"] / (R0 * (0.5 * o["alpha"] + 1))
            sr = 0.5 * so * o["alpha"]
            c0 = (3 - n) / (4 * math.pi * R0 ** (3 - n)) / (math.sqrt(2 * sr * math.pi ** 3) * so)
            f = (0.5 * (1 + torch.erf((R0 - r) / o["smoothingRadius"])) * c0
                 * torch.exp(-u * u / (2 * sr) - l2 / so) * r ** -n)
            return torch.clamp(f, min=1e-200)
        a = o["R0"]
        if t == "Plummer":
            e = 1 / torch.sqrt(r * r + a * a) - 0.5 * (u * u + l2)
            return torch.clamp(2 * e, min=0.0) ** 3.5 * (3 / (7 * math.pi ** 3))
        e = 1 / (a + r) - 0.5 * (u * u + l2)
        q = torch.sqrt(torch.clamp(a * e, min=0.0))
        q2 = q * q
        f = ((1 - q2) ** -2.5 / (8 * math.sqrt(2) * (math.pi * math.sqrt(a)) ** 3)
             * (3 * torch.asin(q) + q * torch.sqrt(1 - q2) * (1 - 2 * q2)
                * (8 * q2 * q2 - 8 * q2 - 3)))
        return torch.where(e > 0, f, torch.zeros_like(f))

    def initial(self, th=None):
        f = self.profile(self.R[None, None, :], self.U[None, :, None], self.J[:, None, None], th)
        v = self.profile(self.er, self.eu, self.ej, th)
        fac = 1 / self.total(f)
        return f * fac, torch.where(self.tail, torch.zeros_like(v), v) * fac

    def mid(self, f):
        return 0.25 * (f[:, :-1, :-1] + f[:, :-1, 1:] + f[:, 1:, :-1] + f[:, 1:, 1:])

    def total(self, f):
        return torch.einsum("jur,j,u,r->", self.mid(f), self.ct, self.dU[:-1], self.dR[:-1])

    def bins(self, f):
        T = torch.einsum("jur,u,j->r", f, self.bu, self.ct)
        return torch.cat([0.25 * self.dR[:-1] * (T[:-1] + T[1:]), T[:1] * 0])

    def stats(self, f):
        b, m = self.bins(f), self.mid(f)
        w = (self.ct[:, None, None] * self.dU[None, :-1, None]) * self.dR[None, None, :-1]
        um, rm = self.U[:-1] + 0.5 * self.dU[:-1], self.R[:-1] + 0.5 * self.dR[:-1]
        v2 = um[None, :, None] ** 2 + (self.J[:, None, None] / rm[None, None, :]) ** 2
        ek = float((w * 0.5 * m * v2).sum())
        s = float((w * torch.where(m > 0, -m * torch.log(torch.clamp(m, min=1e-300)),
                                   torch.zeros_like(m))).sum())
        before = torch.cumsum(b, 0) - b
        ep = -float((b[:-1] * before[:-1] / (0.5 * (self.R[1:] + self.R[:-1]))).sum())
        return [float(b.sum()), ek + ep, ek, ep, s, float((w * m.abs()).sum()),
                float((w * m * m).sum())]

    def kick(self, f):
        nj, nu, nr = self.shape
        M = torch.cumsum(self.bins(f), 0)
        shift = torch.cat([M[:1] * 0, M[:-1]]) * self.coef
        to = self.U[:, None] + shift[None, :]
        y = (to - self.U[0]) * self.hu
        k = torch.floor(y.detach())
        inside = (to > self.U[0]) & (to < self.U[-1])
        k0 = torch.where(inside, k, torch.zeros_like(k)).long()
        w = _weights(y - k)
        c = torch.nn.functional.pad(torch.matmul(self.Pu, f), (0, 0, 0, 1)).reshape(nj, -1)
        col = torch.arange(nr, device="cuda")[None, :]
        v = sum(w[a] * c[:, (k0 + a) * nr + col] for a in range(4))
        return torch.where(inside, v, torch.zeros_like(v))

    def drift(self, f, vals, nd):
        nj, nu, nr = self.shape
        C = torch.matmul(torch.matmul(self.Pu, f), self.Pr.T)
        C = torch.nn.functional.pad(C, (0, 1, 0, 1))
        new = torch.zeros(nj * nu * nr, dtype=torch.float64, device="cuda")
        new = new.index_put((self.gather,), _taps(C, *self.foot))
        if self.cell.numel():
            tv = torch.zeros(self.cell.numel(), dtype=torch.float64, device="cuda")
            tv = tv.index_put((torch.nonzero(self.tail_ok).reshape(-1),),
                              _taps(C, *self.tail_foot))
            vals = vals.index_put((self.first + (nd + self.n - 1) % self.n,), tv)
            new = new.index_put((self.cell,), vals[self.first + nd % self.n])
        return new.reshape(self.shape), vals

    def step(self, f, vals, nd):
        """(f, chain values, drifts done) after one step."""
        if self.o.get("noLinking"):
            f, vals = self.drift(f, vals, nd)
            nd += 1
        f, vals = self.drift(self.kick(f), vals, nd)
        return f, vals, nd + 1


def _exact_bins(m, case, f, vals):
    """The bins after the steps, with gradients through every step (the state
    kept once per step, the step's own tensors recomputed)."""
    from torch.utils.checkpoint import checkpoint
    for n in range(case["steps"]):
        f, vals, _ = checkpoint(m.step, f, vals, n, use_reentrant=False)
    return m.bins(f)


def exact(case, seed):
    if case["kind"] == "spline":
        data, xx, yy, sl = _spline_inputs(case, seed)
        C = torch.matmul(torch.matmul(_solve_matrix(case["nu"]), _t(data)),
                         _solve_matrix(case["nr"]).T)
        C = torch.nn.functional.pad(C, (0, 1, 0, 1))
        a, b = math.log(0.01), math.log(25.0)
        x = (torch.log(_t(xx)) - a) * ((case["nr"] - 1) / (b - a))
        y = (_t(yy) + 2.0) * ((case["nu"] - 1) / 4.0)
        i, k = torch.trunc(x), torch.trunc(y)
        return _taps(C, torch.as_tensor(sl, device="cuda"), i.long(), x - i, k.long(), y - k)
    opt = _options(case, seed)
    m = _Model(opt)
    if case["kind"] == "run":
        if case["steps"] * m.R.numel() * m.U.numel() * m.J.numel() > MOST_WORK:
            return None
        rows, nd = [], 0
        with torch.no_grad():
            f, vals = m.initial()
            for n in range(case["steps"]):
                f, vals, nd = m.step(f, vals, nd)
                if (n + 1) % case["every"] == 0:
                    rows.append(m.stats(f))
        return dict(f=f, stats=_t(rows))
    if case["kind"] == "adjoint":
        f, vals = (x.detach().requires_grad_() for x in m.initial())
        bins = _exact_bins(m, case, f, vals)
        df, dv = torch.autograd.grad((bins * _t(_dbins(case, seed))).sum(), (f, vals),
                                     allow_unused=True)
        return bins.detach(), df, torch.zeros_like(vals) if dv is None else dv
    th = {k: _t(opt[k]).requires_grad_() for k in ("R0", "alpha", "smoothingRadius")}
    vol = 4 * math.pi / 3 * (m.R[1:] ** 3 - m.R[:-1] ** 3)
    rho = _exact_bins(m, case, *m.initial(th))[:-1] / vol
    grad = torch.autograd.grad((rho * _t(_dbins(case, seed)[:-1])).sum(), list(th.values()))
    return rho.detach(), torch.stack(grad)
