"""What this solver's speed is measured on: the calls a user makes, over the
range of grids and options they are made with.

Five kinds of call, by the case's "kind":

* ``noalloc``: ``step_noalloc`` on a state the caller holds in device memory
  (a pass copies the initial state there and advances it ``steps`` steps;
  the whole state comes back).  Grids of at most 131072 points.
* ``live``: a solve that stays resident and is advanced a few steps at a time
  by a program that looks at the extraction column in between.
* ``solve``: a whole solve as the reference's body() is called: create, the
  trajectory if there is a source, run to the final time, read the waveform
  rows and the samples behind them, destroy.
* ``batch``: requests of uneven grids through the batch engine: submit all,
  advance until done, read every waveform.
* ``serve``: the same with the request mix of the served stream, source-free
  and plunge-driven ones.

Runs are shorter in time than production ones (hundreds to a few thousand
steps instead of up to a hundred thousand); everything per step is as there.
The extraction column lies where a short run already has a signal.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import bh_ringdown_b200 as bhr
from bh_ringdown_b200.genot import transition_plunge

PI = 3.14159265358979  # as the reference spells it (HighOrder/parm.h:12)


def listed():
    return [
        # The smallest call: one step of a test-sized grid on the caller's memory; launch latency.
        dict(name="noalloc_256x32", kind="noalloc", N=256, M=32, Xmin=-50.0, Xmax=50.0, m=2, steps=1),
        # An embedding program that advances a small source-free grid between its own work.
        dict(name="noalloc_1024x64", kind="noalloc", N=1024, M=64, Xmin=-100.0, Xmax=300.0, m=2, steps=50),
        # Odd, negative m (zero pole rows) and extents that no tile count divides evenly.
        dict(name="noalloc_1216x80_odd", kind="noalloc", N=1216, M=80, Xmin=-100.0, Xmax=300.0, m=-3, steps=20),
        # A monitoring loop over a resident solve of the served stream's smallest grid.
        dict(name="live_2048x64", kind="live", N=2048, M=64, Xmin=-100.0, Xmax=300.0, m=2, steps=16),
        # The plain source-free evolution (1024 x 64 on [-100, 300]) as a whole solve.
        dict(name="solve_1024x64", kind="solve", N=1024, M=64, Xmin=-100.0, Xmax=300.0, m=2, steps=2600,
             x_ext=60.0, precision="fp64", integrator="ssprk3", source=False),
        # Classical RK4, which the configurations name, on a middle grid.
        dict(name="solve_4096x128_rk4", kind="solve", N=4096, M=128, Xmin=-100.0, Xmax=300.0, m=3, steps=600,
             x_ext=30.0, precision="fp64", integrator="rk4", source=False),
        # The plunge-driven ringdown, 8192 x 128 on [-200, 600], a = 0.9.
        dict(name="plunge_8192x128", kind="solve", N=8192, M=128, Xmin=-200.0, Xmax=600.0, m=2, steps=1000,
             x_ext=5.0, precision="fp64", integrator="ssprk3", source=True),
        # The same, mixed precision.
        dict(name="plunge_8192x128_mixed", kind="solve", N=8192, M=128, Xmin=-200.0, Xmax=600.0, m=2, steps=1000,
             x_ext=5.0, precision="mixed", integrator="ssprk3", source=True),
        # The reference's own default grid (16000 x 256 on [-50, 50]), an odd mode of its m loop, source-free.
        dict(name="solve_16000x256", kind="solve", N=16000, M=256, Xmin=-50.0, Xmax=50.0, m=1, steps=400,
             x_ext=22.0, precision="fp64", integrator="ssprk3", source=False),
        # The largest grid, plunge-driven: the benchmark's default workload.
        dict(name="plunge_16384x256", kind="solve", N=16384, M=256, Xmin=-200.0, Xmax=600.0, m=2, steps=600,
             x_ext=5.0, precision="fp64", integrator="ssprk3", source=True),
        # Source-free solves of uneven grids advanced together, FP64.
        dict(name="batch_12", kind="batch", precision="fp64", T=2.0,
             grids="2048x64 2048x256 4096x64 4096x128 8192x64 8192x128 16384x64 2048x128 4096x128 4096x256 8192x256 "
                   "16384x128"),
        # The served stream's mix: seven source-free requests and three plunges, mixed precision.
        dict(name="serve_10_mixed", kind="serve", precision="mixed", T=4.0, plunges=3,
             grids="2048x64 4096x80 2048x96 4096x128 2048x112 4096x64 2048x128"),
    ]


MAX_POINT_STEPS = 16384 * 256 * 600  # the largest listed case
SMALL_STEPS = {"noalloc": (1, 64), "live": (1, 64)}


def _log_int(rng, lo, hi, step):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["noalloc", "noalloc", "live", "solve", "solve", "solve", "batch", "serve"])
    m = rng.choice([-3, -2, -1, 1, 2, 3, 4])
    if kind in SMALL_STEPS:
        top = 131072 if kind == "noalloc" else 1 << 20
        M = _log_int(rng, 16, 160, 16)
        N = _log_int(rng, 128, min(8192, top // M // 64 * 64), 64)
        Xmin, Xmax = rng.choice([(-50.0, 50.0), (-100.0, 300.0)])
        return dict(kind=kind, N=N, M=M, Xmin=Xmin, Xmax=Xmax, m=m, steps=_log_int(rng, *SMALL_STEPS[kind], 1))
    if kind == "solve":
        M = _log_int(rng, 32, 256, 16)
        N = _log_int(rng, 512, 16384, 64)
        source = rng.random() < 0.4
        integrator = rng.choice(["ssprk3", "ssprk3", "rk4"])
        precision = rng.choice(["fp64", "mixed"]) if integrator == "ssprk3" else "fp64"
        steps = min(_log_int(rng, 100, 2000, 1), MAX_POINT_STEPS * 2 // 3 // (N * M))
        Xmin, Xmax = (-200.0, 600.0) if source else (-100.0, 300.0)
        return dict(kind=kind, N=N, M=M, Xmin=Xmin, Xmax=Xmax, m=2 if source else m, steps=steps,
                    x_ext=5.0 if source else 25.0, precision=precision, integrator=integrator, source=source)
    if kind == "batch":
        grids = ["%dx%d" % (rng.choice([2048, 4096, 8192, 16384]), rng.choice([64, 128, 256]))
                 for _ in range(rng.randint(3, 12))]
        return dict(kind=kind, precision=rng.choice(["fp64", "mixed"]), T=round(rng.uniform(0.5, 1.2), 3),
                    grids=" ".join(grids))
    grids = ["%dx%d" % (rng.choice([2048, 4096]), rng.choice([64, 80, 96, 112, 128])) for _ in range(rng.randint(2, 14))]
    return dict(kind=kind, precision=rng.choice(["fp64", "mixed"]), T=round(rng.uniform(1.0, 4.0), 3),
                plunges=rng.randint(1, 4), grids=" ".join(grids))


# ---- the inputs: parameters and initial data from the case and the seed --------
def _courant_dt(N, M, Xmin, Xmax, r_min=1.6):
    """The Courant rule 0.25 min(dx, r_min dtheta); r at the inner end is
    the horizon radius to machine precision, taken as 1.6 so that a case's
    step count does not depend on the spin drawn."""
    return 0.25 * min((Xmax - Xmin) / N, r_min * math.pi / M)


def _column(x, N, Xmin, Xmax):
    return min(N - 1, max(0, int(round((x - Xmin) * N / (Xmax - Xmin)))))


def _free(rng, N, M, Xmin, Xmax, m, steps, x_ext=None, precision="fp64", integrator="ssprk3"):
    """A source-free solve of `steps` steps: spin, pulse centre and width drawn."""
    a, width = float(rng.uniform(0.0, 0.95)), float(rng.uniform(1.0, 4.0))
    centre = float(rng.uniform(10.0, 20.0 if Xmax < 100.0 else 40.0)) if x_ext is None else float(
        rng.uniform(18.0, 22.0))
    x_ext = centre + width if x_ext is None else x_ext
    dt = _courant_dt(N, M, Xmin, Xmax)
    return bhr.Params(N=N, M=M, Xmin=Xmin, Xmax=Xmax, a=a, m=float(m), dt=dt, T=(steps + 0.5) * dt, Fr=10,
                      out_start=0.0, ext_col=_column(x_ext, N, Xmin, Xmax), init_kind=bhr.BHR_INIT_GAUSSIAN,
                      init_center=centre, init_width=width, init_ell=float(max(2, abs(m))),
                      precision=bhr.BHR_MIXED if precision == "mixed" else bhr.BHR_FP64,
                      integrator=bhr.BHR_RK4 if integrator == "rk4" else bhr.BHR_SSPRK3)


def _plunge(rng, N, M, Xmin, Xmax, m, steps, x_ext, precision="fp64", integrator="ssprk3"):
    """A plunge-driven solve and its worldline (mass ratio 1e-3, from the ISCO)."""
    a = float(rng.uniform(0.85, 0.92))
    dt = _courant_dt(N, M, Xmin, Xmax, 1.4)
    p = bhr.Params(N=N, M=M, Xmin=Xmin, Xmax=Xmax, a=a, m=float(m), dt=dt, T=(steps + 0.5) * dt, Fr=10, out_start=0.0,
                   ext_col=_column(x_ext, N, Xmin, Xmax),
                   precision=bhr.BHR_MIXED if precision == "mixed" else bhr.BHR_FP64,
                   integrator=bhr.BHR_RK4 if integrator == "rk4" else bhr.BHR_SSPRK3)
    return p, transition_plunge(a, 1e-3, dt / 2.0, p.T)


def _steps_of(N, M, T, Xmin=-100.0, Xmax=300.0):
    return max(1, int(T / _courant_dt(N, M, Xmin, Xmax)))


def _grids(case):
    return [tuple(int(v) for v in g.split("x")) for g in case["grids"].split()]


PLUNGE = (8192, 128, -200.0, 600.0)  # the served stream's plunge grid


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for N, M in _grids(case):
        out.append((_free(rng, N, M, -100.0, 300.0, int(rng.integers(1, 5)), _steps_of(N, M, case["T"]),
                          precision=case["precision"]), None))
    for _ in range(case.get("plunges", 0)):
        out.append(_plunge(rng, *PLUNGE, 2, _steps_of(PLUNGE[0], PLUNGE[1], case["T"], *PLUNGE[2:]), 5.0,
                           precision=case["precision"]))
    return out


def _swsh2(ell, m, theta):
    """The s = -2 spin-weighted spherical harmonic on an array of theta (HighOrder/proj.c:16-35)."""
    f = math.factorial
    acc = np.zeros_like(theta)
    for t in range(max(0, m - 2), min(ell + m, ell - 2) + 1):
        c = (-1) ** t * math.sqrt(f(ell + m) * f(ell - m) * f(ell + 2) * f(ell - 2))
        c /= f(ell + m - t) * f(ell - 2 - t) * f(t) * f(t + 2 - m)
        acc += c * np.cos(theta / 2) ** (2 * ell + m - 2 - 2 * t) * np.sin(theta / 2) ** (2 * t + 2 - m)
    return math.sqrt((2 * ell + 1) / 4.0 / PI) * acc


def _close(u, even):
    """The boundary closure of the planes u[..., M, N] (HighOrder/kern.cu:320-449), in place."""
    M, N = u.shape[-2:]
    for r, r1, r2 in ((2, 3, 4), (1, 2, 3), (M - 3, M - 4, M - 5), (M - 2, M - 3, M - 4), (0, 1, 2), (M - 1, M - 2, M - 3)):
        u[..., r, 3:N - 3] = (4.0 * u[..., r1, 3:N - 3] - u[..., r2, 3:N - 3]) / 3.0 if even else 0.0
    for c, c1, c2 in ((2, 3, 4), (N - 3, N - 4, N - 5), (1, 2, 3), (N - 2, N - 3, N - 4), (0, 1, 2), (N - 1, N - 2, N - 3)):
        u[..., c] = (4.0 * u[..., c1] - u[..., c2]) / 3.0
    return u


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pulse(p):
    """The Gaussian pulse of the parameters as a closed state [4, M, N]."""
    x = p.Xmin + np.arange(p.N) * ((p.Xmax - p.Xmin) / p.N) - p.init_center
    fa = np.exp(-x * x / (2.0 * p.init_width * p.init_width))
    gb = _swsh2(int(p.init_ell), int(p.m), np.arange(p.M) * (PI / p.M))
    u = torch.zeros(4, p.M, p.N, dtype=torch.float64, device=_device())
    u[0] = torch.from_numpy(gb[:, None] * fa[None, :])
    return _close(u, int(p.m) % 2 == 0)


# ---- one pass -----------------------------------------------------------------
def _one_solve(case, seed):
    rng = np.random.default_rng(seed)
    make = _plunge if case["source"] else _free
    got = make(rng, case["N"], case["M"], case["Xmin"], case["Xmax"], case["m"], case["steps"], case["x_ext"],
               precision=case["precision"], integrator=case["integrator"])
    return got if case["source"] else (got, None)


def _small(case, seed):
    return _free(np.random.default_rng(seed), case["N"], case["M"], case["Xmin"], case["Xmax"], case["m"], case["steps"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "noalloc":
        p = _small(case, seed)
        u0 = _pulse(p)
        return dict(kind=kind, params=p, steps=case["steps"], start=u0, work=torch.empty_like(u0))
    if kind == "live":
        p = _small(case, seed)
        p.T, p.Fr = 1000.0, 50  # it goes on long after the first calls
        return dict(kind=kind, steps=case["steps"], solver=bhr.Solver(p))
    if kind == "solve":
        p, rows = _one_solve(case, seed)
        return dict(kind=kind, params=p, rows=rows)
    return dict(kind=kind, requests=_requests(case, seed))


def run(state):
    kind = state["kind"]
    if kind == "noalloc":
        state["work"].copy_(state["start"])
        bhr.step_noalloc(state["params"], state["work"].data_ptr(), state["steps"],
                         torch.cuda.current_stream().cuda_stream)
        return state["work"]
    if kind == "live":
        state["solver"].step(state["steps"])
        return state["solver"].get_extraction()
    if kind == "solve":
        with bhr.Solver(state["params"]) as s:
            if state["rows"] is not None:
                s.set_trajectory(state["rows"])
            s.run()
            return [list(s.waveform()), list(s.psi_samples())]
    with bhr.Engine() as e:
        ids = [e.submit(p, rows) for p, rows in state["requests"]]
        e.run_all()
        return [list(e.result(i)) for i in ids]


# ---- what a pass cannot do without ---------------------------------------------
FLOPS_PER_POINT_STAGE = 230  # the right-hand side, its coefficients and the stage combination


def work(case):
    """A step reads the state and writes the next one (4 planes of 8 bytes
    each way); the operations are those of its stages."""
    if case["kind"] in ("batch", "serve"):
        points = sum(N * M * _steps_of(N, M, case["T"]) for N, M in _grids(case))
        N, M, Xmin, Xmax = PLUNGE
        points += case.get("plunges", 0) * N * M * _steps_of(N, M, case["T"], Xmin, Xmax)
    else:
        points = case["N"] * case["M"] * case["steps"]
    stages = 4 if case.get("integrator") == "rk4" else 3
    return dict(bytes=64.0 * points, flops=float(FLOPS_PER_POINT_STAGE * stages) * points)


# ---- the same results in 64 bits, from the reference's formulas ------------------
def _radii(p):
    """r(x): Newton's iteration on the Kerr tortoise coordinate of x / Omega,
    from the outer end inwards; from the first point that falls on the
    horizon in 64 bits, the next number above r+."""
    x = p.Xmin + np.arange(p.N) * ((p.Xmax - p.Xmin) / p.N)
    rin, R = p.Xmin + (p.Xmax - p.Xmin) * 0.64, p.Xmax + 1e-6
    tx = np.where(x < rin, x, x / (1.0 - ((x - rin) / (R - rin)) ** 4))
    mass, a = p.mass, p.a
    root = math.sqrt(mass * mass - a * a)
    rp, rm = mass + root, mass - root
    r = np.full(p.N, np.nextafter(rp, np.inf))
    old = float(tx[-1])
    for i in range(p.N - 1, -1, -1):
        while True:
            t = old + (rp * rp + a * a) / (rp - rm) * math.log(old / rp - 1.0)
            t -= (rm * rm + a * a) / (rp - rm) * math.log(old / rm - 1.0) if a else 0.0
            new = old + (float(tx[i]) - t) * (old * old + a * a - 2.0 * mass * old) / (old * old + a * a)
            if not new > rp:
                return x, r
            done = abs(new - old) / old <= 1e-12
            old = new
            if done:
                break
        r[i] = new
    return x, r


class _Exact:
    """The evolution in plain torch, 64 bits (HighOrder/kern.cu:84-753)."""

    def __init__(self, p):
        self.p = p
        M, a, em, mass = p.M, p.a, p.m, p.mass
        x, r = _radii(p)
        self.r = r
        self.theta = np.arange(M) * (PI / M)
        rin, R = p.Xmin + (p.Xmax - p.Xmin) * 0.64, p.Xmax + 1e-6
        L = R - rin
        s = np.maximum(x - rin, 0.0)
        Om, O1, O2 = 1.0 - (s / L) ** 4, -4.0 * s ** 3 / L ** 4, -12.0 * s ** 2 / L ** 4
        cL, e = Om - x * O1, Om * r
        Sg, Dt = e ** 2 + Om ** 2 * a * a, e ** 2 - 2.0 * e * mass * Om + Om ** 2 * a * a
        y = self.theta[3:M - 3, None]
        sn, cs = np.sin(y), np.cos(y)
        bir = -(2.0 * cL - Om ** 2) * Sg ** 2 / cL ** 2 + a * a * Dt * sn ** 2
        At, Ar = 2.0 * (cL - Om ** 2) * Sg ** 2 / (bir * cL ** 2), -Om ** 2 * Sg ** 2 / (bir * cL ** 2)
        btr = -Om * (e ** 3 * (4.0 * cL ** 2 * (e - 3.0 * mass * Om) + 2.0 * cL * e ** 2 * O1 + e ** 2 * Om * O2 * x)
                     + 2.0 * e * a ** 2 * (cL ** 2 * Om ** 2 * (5.0 * e - 4.0 * mass * Om)
                                           - 3.0 * cL ** 3 * (e - 2.0 * mass * Om) + 2.0 * cL * e ** 2 * Om ** 2 * O1
                                           + e ** 2 * Om ** 3 * O2 * x)
                     + a ** 4 * (-6.0 * cL ** 3 * Om ** 2 + 6.0 * cL ** 2 * Om ** 4 + 2.0 * cL * e * Om ** 4 * O1
                                 + e * Om ** 5 * O2 * x)) / (bir * cL ** 3 * e)
        h = 2.0 * Om * O1 - 2.0 * O1 ** 2 * x + Om * O2 * x
        brr = -Om * (e ** 5 * h + 2.0 * e ** 3 * Om ** 2 * h * a ** 2
                     + Om ** 4 * a ** 4 * (6.0 * Om ** 2 + 2.0 * O1 ** 2 * x * (-e + 3.0 * x)
                                           + Om * (2.0 * e * O1 - 12.0 * O1 * x + e * O2 * x))
                     + 2.0 * cL ** 2 * e * (2.0 * e ** 3 - 6.0 * e ** 2 * mass * Om + 5.0 * e * Om ** 2 * a ** 2
                                            - 4.0 * mass * Om ** 3 * a ** 2)) / (bir * cL ** 3 * e)
        bti = 2.0 * a * (em * (-Om ** 2 * Sg + cL * (e ** 2 + 2.0 * e * mass * Om + Om ** 2 * a * a))
                         - 2.0 * cL * Dt * cs) / (bir * cL)
        bri = -2.0 * em * Om ** 2 * a * Sg / (bir * cL)
        cre = Dt * (2.0 * e ** 2 + 6.0 * e * mass * Om - 6.0 * Om ** 2 * a * a
                    + e ** 2 * (2.0 * cs - em) ** 2 / sn ** 2) / (bir * e ** 2)
        cim = 2.0 * em * Om * a * (e ** 2 + 2.0 * e * mass * Om - 3.0 * Om ** 2 * a * a) / (bir * e)
        bb = -(At + np.sqrt(At * At + 4.0 * Ar)) / 2.0
        dev = _device()
        dx, dth = (p.Xmax - p.Xmin) / p.N, PI / M
        self.cx, self.cy, self.cyy = 0.016666666666667 / dx, 1.0 / (60.0 * dth), 1.0 / (180.0 * dth * dth)
        self.cko = 0.1 * 0.0625 / p.dt

        def plane(v):
            return torch.from_numpy(np.ascontiguousarray(np.broadcast_to(v, bb.shape)[:, 3:-3])).to(dev)

        db = np.zeros_like(bb)
        db[:, 3:-3] = (45.0 * (bb[:, 4:-2] - bb[:, 2:-4]) - 9.0 * (bb[:, 5:-1] - bb[:, 1:-5]) + bb[:, 6:] - bb[:, :-6])
        self.bb, self.ee, self.cc = plane(bb), plane(At + bb), plane(-Dt / bir)
        self.d = torch.complex(plane(brr - bb * btr - db * self.cx * (At + bb)), plane(bri - bb * bti))
        self.a = torch.complex(plane(-btr), plane(-bti))
        self.v = torch.complex(plane(-cre), plane(-cim))
        self.ctan = torch.from_numpy(np.tan(0.5 * PI - y)).to(dev)
        self.even = int(em) % 2 == 0

    def rhs(self, u):
        """d/dt of the closed complex planes u[2, M, N] on the interior."""
        q, p = u
        N = q.shape[1]
        row = [q[k:k + q.shape[0] - 6, 3:-3] for k in range(7)]
        y1 = 45.0 * (row[4] - row[2]) - 9.0 * (row[5] - row[1]) + row[6] - row[0]
        y2 = 2.0 * (row[6] + row[0]) - 27.0 * (row[5] + row[1]) + 270.0 * (row[4] + row[2]) - 490.0 * row[3]
        ll = y2 * self.cyy + self.ctan * (y1 * self.cy)
        c = u[:, 3:-3]
        col = [c[..., k:k + N - 6] for k in range(7)]
        x1 = (45.0 * (col[4] - col[2]) - 9.0 * (col[5] - col[1]) + col[6] - col[0]) * self.cx
        ko = torch.zeros_like(x1)
        w = [c[..., k:k + N - 8] for k in range(9)]
        ko[..., 1:-1] = (w[8] + w[0] - 8.0 * (w[7] + w[1]) + 28.0 * (w[6] + w[2]) - 56.0 * (w[5] + w[3])
                         + 70.0 * w[4]) * self.cko
        q0, p0 = col[3]
        return torch.stack((p0 - self.bb * x1[0] - ko[0],
                            self.ee * x1[1] - ko[1] + self.cc * ll + self.d * x1[0] - self.a * p0 - self.v * q0))

    def step(self, u):
        dt = self.p.dt

        def closed(inner):
            out = torch.zeros_like(u)
            out[:, 3:-3, 3:-3] = inner
            return _close(out, self.even)

        i = u[:, 3:-3, 3:-3]
        if self.p.integrator == bhr.BHR_RK4:
            k1 = self.rhs(u)
            k2 = self.rhs(closed(i + 0.5 * dt * k1))
            k3 = self.rhs(closed(i + 0.5 * dt * k2))
            k4 = self.rhs(closed(i + dt * k3))
            return closed(i + dt / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4))
        u1 = closed(i + dt * self.rhs(u))
        u2 = closed(0.75 * i + 0.25 * (u1[:, 3:-3, 3:-3] + dt * self.rhs(u1)))
        return closed((i + 2.0 * (u2[:, 3:-3, 3:-3] + dt * self.rhs(u2))) / 3.0)

    def weights(self):
        """Boole's rule times the harmonics for l = |m| .. |m|+6, and the dE/dt weights (HighOrder/body.cu:168-212)."""
        p, M, mabs, dth = self.p, self.p.M, abs(int(self.p.m)), PI / self.p.M
        th = np.arange(M + 1) * dth
        w = np.zeros(M + 1)
        for i in range(M // 4):
            w[4 * i:4 * i + 5] += np.array([7.0, 32.0, 12.0, 32.0, 7.0]) * 2.0 / 45.0
        proj = np.stack([w * 4.0 * PI * np.sin(th) * dth * _swsh2(l, int(p.m), th)
                         for l in range(mabs, mabs + 7)])
        proj[:, M - 1] += proj[:, M]
        rr = self.r[-1]
        rho2 = rr * rr + (p.a * np.cos(self.theta)) ** 2
        return proj[:, :M], 0.5 * dth * np.sin(self.theta) * rr ** 8 / rho2 ** 4

    def evolve(self, steps):
        """(columns of psi after each step [steps, M], the final closed state)."""
        s = _pulse(self.p)
        u = torch.stack((torch.complex(s[0], s[1]), torch.complex(s[2], s[3])))
        got = []
        for _ in range(steps):
            u = self.step(u)
            got.append(u[0, :, self.p.ext_col].clone())
        return torch.stack(got).cpu().numpy(), u

    def waveform(self, steps):
        """What waveform() and psi_samples() return: t, h, dE/dt and the samples, every Fr steps."""
        psi, _ = self.evolve(steps)
        p, rows = self.p, np.arange(0, steps, self.p.Fr)
        first = np.cumsum(psi, axis=0) * p.dt
        second = np.cumsum(first, axis=0) * p.dt
        proj, flux = self.weights()
        h = np.empty((len(rows), 14))
        h[:, 0::2] = second[rows].real @ proj.T
        h[:, 1::2] = -second[rows].imag @ proj.T
        dedt = (np.abs(first[rows]) ** 2) @ flux
        timer = np.concatenate(([0.0], np.cumsum(np.full(steps, p.dt))))[rows]
        return [timer - p.Xmax, h, dedt], [np.ascontiguousarray(psi[rows].real), np.ascontiguousarray(psi[rows].imag)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("noalloc", "live"):
        s = _Exact(_small(case, seed))
        psi, u = s.evolve(case["steps"])
        if kind == "noalloc":
            return torch.stack((u[0].real, u[0].imag, u[1].real, u[1].imag))
        first = np.cumsum(psi, axis=0) * s.p.dt
        second = np.sum(first, axis=0) * s.p.dt
        return [np.ascontiguousarray(v) for z in (psi[-1], first[-1], second) for v in (z.real, z.imag)]
    if kind == "solve":
        if case["source"]:
            return None  # the source's coefficients have no short form to restate here
        return list(_Exact(_one_solve(case, seed)[0]).waveform(case["steps"]))
    out = []
    for p, rows in _requests(case, seed):
        out.append(None if rows is not None else _Exact(p).waveform(int(p.T / p.dt))[0])
    return out
