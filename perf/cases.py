"""What a user of this framework runs, as timed cases.

The framework advances flows around immersed bodies (`solve_` with a `Solver`, or an `Ensemble` of
them) in two precisions, "fp64" (the default) and "mixed", and offers its stream-function
operators on device arrays (include/ibgb300_ops.h).  The cases are those calls:

* ``solve``: a stretch of a run: `steps` time steps through `solve_`, the C_D / C_L of every step,
  and the state the program keeps at the end of the stretch (a snapshot in pinned host memory).
  CNAB in both precisions, RKC, one body or several, bodies at rest or moving (Schur-
  preconditioned CG); with a per-step callback (a monitor that reads the forces as they come) or
  without (the steps run as one batch).
* ``ensemble``: a parameter sweep: several members stepped by one `Ensemble`.
* ``poisson``, ``vort2flux``: a program that keeps its own arrays on the GPU and calls the
  operators: the Poisson solve on a batch of fields, vorticity to stream function and flux.

An FP64 run returns the state a restart needs (circulation, flux, stream function, nonlinear
history) and its force coefficients in FP64.  A mixed run returns the circulation (what its flux and
stream function are computed from) in FP64, and its force coefficients, which carry about seven
digits by that mode's contract, in single precision.
"""
import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import package

ib = package()


# --------------------------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest grid of the repository's ensembles, stepped one by one with its forces read
        # after each step: latency and launches are all of it
        {"name": "step_128_fp64", "kind": "solve", "scheme": "cnab", "precision": "fp64", "nx": 128, "ny": 128,
         "levels": 3, "h": 4 / 128, "x0": -1.5, "y0": -2.0, "re": 100.0, "dt": 0.2 * 4 / 128,
         "bodies": "ellipse 0 0 1.0 0.5 20 1.0", "steps": 1, "callback": True},
        # the cylinder workload (Re 100, 200 x 200, 5 levels) in the default precision, forces
        # monitored at every step; a grid that is no power of two
        {"name": "cylinder_200_fp64", "kind": "solve", "scheme": "cnab", "precision": "fp64", "nx": 200, "ny": 200,
         "levels": 5, "h": 0.02, "x0": -1.0, "y0": -2.0, "re": 100.0, "dt": 0.004,
         "bodies": "cylinder 0 0 1.0 157", "steps": 20, "callback": True},
        # the explicit scheme at an ordinary size
        {"name": "rkc_384x256_fp64", "kind": "solve", "scheme": "rkc", "precision": "fp64", "nx": 384, "ny": 256,
         "levels": 4, "h": 4 / 384, "x0": -1.5, "y0": -128 * 4 / 384, "re": 200.0, "dt": 0.2 * 4 / 384,
         "bodies": "ellipse 0 0 1.0 0.4 15 1.0", "steps": 10, "callback": False},
        # the two-body workload (1024 x 1024, 4 levels) in FP64
        {"name": "two_body_1024_fp64", "kind": "solve", "scheme": "cnab", "precision": "fp64", "nx": 1024, "ny": 1024,
         "levels": 4, "h": 0.005, "x0": -1.5, "y0": -2.56, "re": 200.0, "dt": 0.001,
         "bodies": "cylinder 0 0.8 1.0 629; plate 0 -0.8 1.0 20 201", "steps": 8, "callback": False},
        # a small mixed run with a per-step monitor
        {"name": "step_256x192_mixed", "kind": "solve", "scheme": "cnab", "precision": "mixed", "nx": 256, "ny": 192,
         "levels": 3, "h": 4 / 256, "x0": -1.5, "y0": -96 * 4 / 256, "re": 150.0, "dt": 0.2 * 4 / 256,
         "bodies": "ellipse 0 0 1.0 0.3 10 1.0", "steps": 10, "callback": True},
        # the two-body workload in mixed precision, the benchmark's configuration
        {"name": "two_body_1024_mixed", "kind": "solve", "scheme": "cnab", "precision": "mixed", "nx": 1024,
         "ny": 1024, "levels": 4, "h": 0.005, "x0": -1.5, "y0": -2.56, "re": 200.0, "dt": 0.001,
         "bodies": "cylinder 0 0.8 1.0 629; plate 0 -0.8 1.0 20 201", "steps": 20, "callback": False},
        # the largest grid, five levels, mixed (the four-cylinder workload's grid with one plate)
        {"name": "plate_2048_mixed", "kind": "solve", "scheme": "cnab", "precision": "mixed", "nx": 2048, "ny": 2048,
         "levels": 5, "h": 0.0025, "x0": -2.0, "y0": -2.56, "re": 150.0, "dt": 0.0005,
         "bodies": "plate 0 0 0.5 15 201", "steps": 10, "callback": False},
        # the heaving and pitching plate: weights rebuilt and CG every step
        {"name": "moving_plate_mixed", "kind": "solve", "scheme": "cnab", "precision": "mixed", "nx": 768, "ny": 512,
         "levels": 4, "h": 0.005, "x0": -1.0, "y0": -1.28, "re": 1000.0, "dt": 0.0005,
         "bodies": "moving 0.2 0.5 30 1.0 201", "steps": 4, "callback": False},
        # a sweep of eight static members over the repository's ensemble shapes
        {"name": "ensemble_8_mixed", "kind": "ensemble", "precision": "mixed", "members": 8, "pick": 0, "steps": 8},
        # one small Poisson solve on the device: a call's fixed cost
        {"name": "poisson_64x48", "kind": "poisson", "nx": 64, "ny": 48, "batch": 1},
        # the largest grid, a batch of fields
        {"name": "poisson_2048_batch2", "kind": "poisson", "nx": 2048, "ny": 2048, "batch": 2},
        # vorticity to flux on a ragged grid (600 = 8*3*25, 400 = 16*25)
        {"name": "vort2flux_600x400", "kind": "vort2flux", "nx": 600, "ny": 400, "levels": 4},
    ]


def _rest(m):
    for p in (2, 3, 5):
        while m % p == 0:
            m //= p
    return m


#: axis lengths the transforms accept (multiples of 4 with n/2 a product of 2, 3 and 5), 64 to 2048
AXES = [n for n in range(64, 2049, 4) if _rest(n // 2) == 1]


def _axis(rng, lo, hi):
    """An accepted axis length, spread over the logarithm of [lo, hi]."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(AXES, key=lambda n: abs(math.log(n / want)))


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "mixed", "mixed", "rkc", "moving", "ensemble", "poisson", "vort2flux"])
    if kind == "poisson":
        return {"kind": "poisson", "nx": _axis(rng, 64, 2048), "ny": _axis(rng, 64, 2048),
                "batch": rng.choice([1, 1, 2, 3])}
    if kind == "vort2flux":
        return {"kind": "vort2flux", "nx": _axis(rng, 64, 1200), "ny": _axis(rng, 64, 1200),
                "levels": rng.randint(2, 5)}
    if kind == "ensemble":
        return {"kind": "ensemble", "precision": "mixed", "members": rng.randint(3, 8),
                "pick": rng.randint(1, 10 ** 6), "steps": rng.randint(2, 8)}
    if kind == "moving":
        nx = _axis(rng, 256, 768)
        ny = _axis(rng, 0.6 * nx, 0.8 * nx)
        h = 3.84 / nx
        n = int(1.0 / h) + 1
        return {"kind": "solve", "scheme": "cnab", "precision": "mixed", "nx": nx, "ny": ny,
                "levels": rng.randint(3, 4), "h": h, "x0": -1.0, "y0": -0.5 * ny * h, "re": 1000.0, "dt": 0.1 * h,
                "bodies": "moving 0.2 0.25 %d 1.0 %d" % (rng.randint(5, 25), n), "steps": rng.randint(2, 4),
                "callback": False}
    top = {"fp64": 1024, "mixed": 2048, "rkc": 512}[kind]
    nx = _axis(rng, 128, top)
    ny = _axis(rng, max(96, nx / 2), min(top, nx * 1.2))
    h = 4.0 / nx
    # the body's chord keeps its points (about one per cell) at four hundred or fewer
    chord = min(1.0, 130 * h)
    return {"kind": "solve", "scheme": "rkc" if kind == "rkc" else "cnab",
            "precision": "mixed" if kind == "mixed" else "fp64", "nx": nx, "ny": ny, "levels": rng.randint(2, 5),
            "h": h, "x0": -1.5, "y0": -0.5 * ny * h, "re": float(round(math.exp(rng.uniform(math.log(50), math.log(500))))),
            "dt": 0.2 * h, "bodies": "ellipse 0 0 %.4f %.2f %.1f 1.0" % (chord, rng.uniform(0.2, 1.0), rng.uniform(0, 40)),
            "steps": rng.randint(1, 8), "callback": rng.random() < 0.5}


# --------------------------------------------------------------------------------------------
# geometry
# --------------------------------------------------------------------------------------------
def _bodies(text, h):
    """[(points (n, 2), ds (n,), motion or None)] of a case's bodies."""
    out = []
    for part in text.split(";"):
        word, *v = part.split()
        v = [float(x) for x in v]
        if word == "cylinder":
            x, y, d, n = v
            t = 2 * math.pi * np.arange(int(n)) / int(n)
            xb, ds, motion = np.stack([x + d / 2 * np.cos(t), y + d / 2 * np.sin(t)], 1), math.pi * d / n, None
        elif word == "plate":
            x, y, c, a, n = v
            s, a = np.linspace(-c / 2, c / 2, int(n)), math.radians(a)
            xb, ds, motion = np.stack([x + s * math.cos(a), y - s * math.sin(a)], 1), c / (n - 1), None
        elif word == "ellipse":
            x, y, c, aspect, a, spacing = v
            th, a = np.linspace(0, 2 * math.pi, 4097), math.radians(a)
            ex, ey = c / 2 * np.cos(th), aspect * c / 2 * np.sin(th)
            arc = np.concatenate([[0.0], np.cumsum(np.hypot(np.diff(ex), np.diff(ey)))])
            n = max(8, int(round(arc[-1] / (spacing * h))))
            at = np.arange(n) * arc[-1] / n
            px, py = np.interp(at, arc, ex), np.interp(at, arc, ey)
            xb = np.stack([x + math.cos(a) * px + math.sin(a) * py, y - math.sin(a) * px + math.cos(a) * py], 1)
            ds, motion = arc[-1] / n, None
        else:  # moving: heave amplitude v[1] at frequency v[0], pitch v[2] degrees about the quarter chord
            f, heave, pitch, c, n = v
            xb, ds = np.stack([np.linspace(-0.25 * c, 0.75 * c, int(n)), np.zeros(int(n))], 1), c / (n - 1)
            motion = (2 * math.pi * f, heave, math.radians(pitch))
        out.append((xb, np.full(len(xb), ds), motion))
    return out


def _kinematics(motion, t):
    """r0, v0, theta, Omega of a heaving and pitching body."""
    w, a, p = motion
    return ((0.0, a * math.sin(w * t)), (0.0, a * w * math.cos(w * t)),
            p * math.sin(w * t + math.pi / 2), p * w * math.cos(w * t + math.pi / 2))


def _frame(motion):
    if motion is None:
        return ib.GridFrame()
    return ib.RelativeFrame(ib.GridFrame(), r=lambda t: _kinematics(motion, t)[0], v=lambda t: _kinematics(motion, t)[1],
                            theta=lambda t: _kinematics(motion, t)[2], omega=lambda t: _kinematics(motion, t)[3])


def _noise(nx, ny, levels, h, seed):
    """The workloads' initial circulation: vorticity noise of amplitude 1e-4 on the finest level."""
    g = np.zeros((levels, (nx - 1) * (ny - 1)))
    g[0] = 1e-4 * h * h * np.random.Generator(np.random.PCG64(seed)).standard_normal((nx - 1) * (ny - 1))
    return g


def _members(case):
    """The members of an ensemble case, as solve cases of the repository's ensemble shapes."""
    r = np.random.default_rng(case["pick"])
    grids = [(128, 128), (256, 256), (384, 256), (512, 512)]
    out = []
    for _ in range(case["members"]):
        nx, ny = grids[r.integers(4)]
        h = 4.0 / nx
        out.append({"kind": "solve", "scheme": "cnab", "precision": case["precision"], "nx": nx, "ny": ny,
                    "levels": int(r.integers(3, 6)), "h": h, "x0": -1.5, "y0": -0.5 * ny * h,
                    "re": float(np.exp(r.uniform(math.log(50), math.log(500)))), "dt": 0.2 * h,
                    "bodies": "ellipse 0 0 1.0 %r %r 1.0" % (float(r.uniform(0.2, 1.0)), float(r.uniform(0, 40))),
                    "steps": case["steps"], "callback": False})
    return out


#: steps a moving case has behind it when the timed stretch begins (its first two steps and first
#: preconditioner are set-up of the run)
MOVING_STEPS = 3


# --------------------------------------------------------------------------------------------
# prepare and run
# --------------------------------------------------------------------------------------------
def _grid(case):
    base = ib.UniformGrid(case["h"], (case["x0"], case["x0"] + case["nx"] * case["h"]),
                          (case["y0"], case["y0"] + case["ny"] * case["h"]))
    assert (base.nx, base.ny) == (case["nx"], case["ny"])
    return ib.MultiLevel(base, case["levels"])


class Run:
    """A run in progress: problem, state, solver and the program's snapshot buffers."""

    def __init__(self, case, seed):
        self.case, self.dt, self.t = case, case["dt"], 0.0
        bodies = [ib.RigidBody(_frame(m), xb, ds) for xb, ds, m in _bodies(case["bodies"], case["h"])]
        scheme = ib.SchemeRKC(self.dt) if case["scheme"] == "rkc" else ib.SchemeCNAB(self.dt)
        self.prob = ib.Problem(ib.StreamFcnFluid(_grid(case), (1.0, 0.0), case["re"]), ib.BodyGroup(*bodies), scheme)
        self.state = ib.initstate(self.prob)
        self.state.qty.gamma[:] = _noise(case["nx"], case["ny"], case["levels"], case["h"], seed)
        self.solver = ib.initsolver(self.prob, self.state, precision=case["precision"])
        self.solver.vort2flux(self.state)
        d, L = self.prob.fluid.domain, case["levels"]
        keep = ["gamma"]
        if case["precision"] == "fp64":
            keep = ["gamma", "q", "psi"] + (["nonlin"] if case["scheme"] == "cnab" else [])
        size = {"gamma": (L, d.ngamma), "q": (L, d.nq), "psi": (L, d.ngamma), "nonlin": (L, d.ngamma)}
        self.kept = {k: torch.empty(size[k], dtype=torch.float64, pin_memory=True) for k in keep}
        if self.solver.moving:
            self.solver.set_cg_options(tol=1e-10, warm_start="extrapolate")
            self.solver.set_cg_preconditioner("schur_ref", refresh_steps=20)
            self.stretch(MOVING_STEPS, False)

    def stretch(self, steps, callback):
        """`steps` steps; the (C_D, C_L) of every body at each of them."""
        tlims = (self.t, self.t + (steps - 0.75) * self.dt)
        self.t += steps * self.dt
        if callback:
            got, = ib.solve_(self.state, self.prob, tlims, solver=self.solver,
                             save=(ib.each_timestep(lambda s: [(b.CD, b.CL) for b in s.qty.stress]),))
            return np.array(got).transpose(0, 2, 1)
        ib.solve_(self.state, self.prob, tlims, solver=self.solver)
        return np.stack(self.solver.force_history(steps), 1)

    def snapshot(self):
        """The kept fields from the handle into the program's buffers (ib_get_state)."""
        p = {k: ctypes.cast(v.data_ptr(), ctypes.POINTER(ctypes.c_double)) for k, v in self.kept.items()}
        st = self.solver.lib.ib_get_state(self.solver.handle, p.get("gamma"), p.get("q"), p.get("psi"), None,
                                          p.get("nonlin"), None, None)
        assert st == 0, st
        return self.kept

    def result(self, forces):
        f = forces if self.case["precision"] == "fp64" else forces.astype(np.float32)
        return {"forces": f, **self.snapshot()}


class Operator:
    """A handle whose operators a program calls on its own device arrays."""

    def __init__(self, case, seed):
        nx, ny = case["nx"], case["ny"]
        L = case.get("levels", 1)
        grid = dict(case, h=4.0 / nx, x0=-2.0, y0=-2.0 * ny / nx, levels=L)
        self.prob = ib.Problem(ib.StreamFcnFluid(_grid(grid), (1.0, 0.0), 100.0), ib.BodyGroup(), ib.SchemeCNAB(0.01))
        self.solver = ib.initsolver(self.prob, ib.initstate(self.prob))
        d = self.prob.fluid.domain
        self.x = _fields(case, seed)
        self.out = [torch.empty_like(self.x)]
        if case["kind"] == "vort2flux":
            self.out.append(torch.empty((L, d.nq), dtype=torch.float64, device="cuda"))
        self.args = [ctypes.c_void_p(a.data_ptr()) for a in (self.x, *self.out)]


def _fields(case, seed):
    """Circulations on the device: a few vortices of different cores and signs over weak noise (per
    batch entry, or on the finest level with the coarser levels' own far fields)."""
    nx, ny = case["nx"], case["ny"]
    n = case.get("batch", case.get("levels"))
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kw = {"generator": gen, "device": "cuda", "dtype": torch.float64}
    x = torch.arange(1, nx, device="cuda", dtype=torch.float64) / nx
    y = torch.arange(1, ny, device="cuda", dtype=torch.float64) / ny
    f = 1e-6 * torch.randn((n, ny - 1, nx - 1), **kw)
    for _ in range(4):
        c, w, a = torch.rand((2, n, 1, 1), **kw), 0.01 + 0.1 * torch.rand((n, 1, 1), **kw), torch.randn((n, 1, 1), **kw)
        f += a * torch.exp(-((x[None, None, :] - c[0]) ** 2 + (y[None, :, None] - c[1]) ** 2) / w ** 2)
    return f.reshape(n, -1)


def prepare(case, seed):
    if case["kind"] == "solve":
        return Run(case, seed)
    if case["kind"] == "ensemble":
        runs = [Run(m, seed + k) for k, m in enumerate(_members(case))]
        return {"case": case, "runs": runs, "ensemble": ib.Ensemble([r.solver for r in runs]), "step": 0}
    return {"case": case, "op": Operator(case, seed)}


def run(state):
    if isinstance(state, Run):
        return state.result(state.stretch(state.case["steps"], state.case["callback"]))
    case = state["case"]
    if case["kind"] == "ensemble":
        runs, k, n = state["runs"], state["step"], case["steps"]
        ts = (k + np.arange(n))[:, None] * np.array([r.dt for r in runs])[None, :]
        state["ensemble"].advance_n(ts)
        state["step"] = k + n
        return [r.result(np.stack(r.solver.force_history(n), 1)) for r in runs]
    op = state["op"]
    lib, h = op.solver.lib, op.solver.handle
    if case["kind"] == "poisson":
        st = lib.ib_op_laplacian_inv(h, case["batch"], *op.args)
        assert st == 0, st
        return op.out[0]
    st = lib.ib_op_vort2flux(h, *op.args)
    assert st == 0, st
    return [op.x, *op.out]


# --------------------------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------------------------
def _solve_flops(nx, ny):
    """A Poisson solve: two sine transforms per axis, 2.5 n log2 n operations a line."""
    return 2 * 2.5 * nx * ny * (math.log2(nx) + math.log2(ny))


def work(case):
    if case["kind"] == "ensemble":
        w = [work(m) for m in _members(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    nx, ny = case["nx"], case["ny"]
    ng, nq = (nx - 1) * (ny - 1), (nx + 1) * ny + nx * (ny + 1)
    if case["kind"] == "poisson":
        return {"bytes": 16.0 * case["batch"] * ng, "flops": case["batch"] * _solve_flops(nx, ny)}
    L = case["levels"]
    if case["kind"] == "vort2flux":
        return {"bytes": 8.0 * L * (2 * ng + nq), "flops": L * (_solve_flops(nx, ny) + 12 * ng)}
    # a step reads and writes the state once (circulation, two histories, flux, stream function) and
    # applies the Schur inverse; solves: L trial + 1 projection + 2 L Vort2Flux (RKC: (s + 1) L)
    nb = sum(len(b[0]) for b in _bodies(case["bodies"], case["h"]))
    solves = 3 * L + 1
    if case["scheme"] == "rkc":
        solves = (_rkc_stages(case) + 1) * L
    step = {"bytes": 8.0 * L * (5 * ng + 2 * nq) + 8.0 * (2 * nb) ** 2,
            "flops": solves * _solve_flops(nx, ny) + 60.0 * L * ng + 2.0 * (2 * nb) ** 2}
    out = 8.0 * L * ng if case["precision"] == "mixed" else 8.0 * L * (3 * ng + nq)
    return {"bytes": case["steps"] * step["bytes"] + out, "flops": case["steps"] * step["flops"]}


# --------------------------------------------------------------------------------------------
# exact: the same calls in plain FP64 torch
# --------------------------------------------------------------------------------------------
def _rkc_coefficients(S):
    """mu, nu, mu~, gamma~ (from index 1) and the stability interval of the damped second-order
    Runge-Kutta-Chebyshev method (Sommeijer, Shampine and Verwer 1998)."""
    w0 = 1 + (2 / 13) / S ** 2
    T, D, E = [1.0, w0], [0.0, 1.0], [0.0, 0.0]
    for j in range(2, S + 1):
        T.append(2 * w0 * T[-1] - T[-2])
        E.append(4 * D[-1] + 2 * w0 * E[-1] - E[-2])
        D.append(2 * T[j - 1] + 2 * w0 * D[-1] - D[-2])
    w1 = D[S] / E[S]
    b = [0.0, 0.0] + [E[j] / D[j] ** 2 for j in range(2, S + 1)]
    b[0] = b[1] = b[2]
    mu, nu, mt, gt = [[0.0] * (S + 1) for _ in range(4)]
    mt[1] = b[1] * w1
    for j in range(2, S + 1):
        mu[j], nu[j], mt[j] = 2 * b[j] * w0 / b[j - 1], -b[j] / b[j - 2], 2 * b[j] * w1 / b[j - 1]
        gt[j] = -(1 - b[j - 1] * T[j - 1]) * mt[j]
    return mu, nu, mt, gt, (w0 + 1) * E[S] / D[S]


def _rkc_stages(case):
    S = 2
    while S < 64 and _rkc_coefficients(S)[4] < 1.5 * case["dt"] * 8 / (case["re"] * case["h"] ** 2):
        S += 1
    return S


def _delta(r):
    """The three-cell smoothed delta function (Yang et al. 2009), times h, at distances r >= 0 in cells;
    the coefficients to ten digits, as the solvers of this family use them."""
    s3 = math.sqrt(3.0)

    def root(x):
        return torch.sqrt(torch.clamp(x, min=0.0))

    def asin(x):
        return torch.asin(torch.clamp(x, -1.0, 1.0))

    a, q = asin(s3 / 2 * (2 * r - 1)), root(1 + 12 * r - 12 * r * r)
    one = (4.166666667e-2 * r ** 4 + (-0.1388888889 + 3.472222222e-2 * q) * r ** 3
           + (-7.121664902e-2 - 5.208333333e-2 * q + 0.2405626122 * a) * r ** 2
           + (-0.2405626122 * a - 0.3792313933 + 0.1012731481 * q) * r
           + 8.0187537413e-2 * a - 4.195601852e-2 * q + 0.6485698427)
    a, q = asin(s3 / 2 * (2 * r - 3)), root(-23 + 36 * r - 12 * r * r)
    two = (-6.25e-2 * r ** 4 + (0.4861111111 - 1.736111111e-2 * q) * r ** 3
           + (-1.143175026 + 7.8125e-2 * q - 0.1202813061 * a) * r ** 2
           + (0.8751991178 + 0.3608439183 * a - 0.1548032407 * q) * r
           - 0.2806563809 * a + 8.22848104e-3 + 0.1150173611 * q)
    a, q = asin(s3 / 2 * (2 * r - 5)), root(-71 + 60 * r - 12 * r * r)
    three = (2.083333333e-2 * r ** 4 + (3.472222222e-3 * q - 0.2638888889) * r ** 3
             + (1.214391675 - 2.604166667e-2 * q + 2.405626122e-2 * a) * r ** 2
             + (-0.1202813061 * a - 2.449273192 + 7.262731481e-2 * q) * r
             + 0.1523563211 * a + 1.843201677 - 7.306134259e-2 * q)
    return torch.where(r <= 1, one, torch.where(r <= 2, two, torch.where(r <= 3, three, torch.zeros_like(r))))


class Plain:
    """The stream-function operators on (..., ny-1, nx-1) arrays and (qx, qy) face arrays."""

    def __init__(self, nx, ny, levels, h=1.0):
        self.nx, self.ny, self.L, self.h = nx, ny, levels, h
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        ci = torch.cos(math.pi * self.arange(1, nx) / nx)
        cj = torch.cos(math.pi * self.arange(1, ny) / ny)
        self.lam = 4.0 - 2.0 * (ci[None, :] + cj[:, None])

    def arange(self, *a):
        return torch.arange(*a, dtype=torch.float64, device=self.dev)

    def dst(self, x):
        z = torch.zeros_like(x[..., :1])
        return -torch.fft.rfft(torch.cat([z, x, z, -x.flip(-1)], -1)).imag[..., 1:x.shape[-1] + 1]

    def solve(self, b, eig):
        """The array with sine coefficients b^ / eig."""
        f = self.dst(self.dst(b).transpose(-1, -2)) / (eig.transpose(-1, -2) * (4 * self.nx * self.ny))
        return self.dst(self.dst(f).transpose(-1, -2))

    def ring(self, r):
        """The next finer level's boundary values: left, right (ny+1 each), bottom, top (nx+1 each)."""
        nx, ny = self.nx, self.ny
        j, i = slice(ny // 4 - 1, 3 * ny // 4), slice(nx // 4 - 1, 3 * nx // 4)
        out = []
        for line in (r[..., j, nx // 4 - 1], r[..., j, 3 * nx // 4 - 1], r[..., ny // 4 - 1, i], r[..., 3 * ny // 4 - 1, i]):
            v = torch.empty(line.shape[:-1] + (2 * line.shape[-1] - 1,), dtype=line.dtype, device=line.device)
            v[..., ::2] = line
            v[..., 1::2] = 0.5 * (line[..., 1:] + line[..., :-1])
            out.append(0.25 * v)
        return out

    def edges(self, r, ring, fac):
        left, right, bottom, top = ring
        r = r.clone()
        r[..., 0, :] += fac * bottom[..., 1:-1]
        r[..., -1, :] += fac * top[..., 1:-1]
        r[..., :, 0] += fac * left[..., 1:-1]
        r[..., :, -1] += fac * right[..., 1:-1]
        return r

    def padded(self, psi, ring):
        p = torch.zeros(psi.shape[:-2] + (self.ny + 1, self.nx + 1), dtype=psi.dtype, device=psi.device)
        p[..., 1:-1, 1:-1] = psi
        if ring is not None:
            p[..., 0, :], p[..., -1, :] = ring[2], ring[3]
            p[..., :, 0], p[..., :, -1] = ring[0], ring[1]
        return p

    def curl(self, psi, ring):
        p = self.padded(psi, ring)
        return p[..., 1:, :] - p[..., :-1, :], p[..., :, :-1] - p[..., :, 1:]

    def rot(self, qx, qy):
        return qx[..., :-1, 1:-1] - qx[..., 1:, 1:-1] + qy[..., 1:-1, 1:] - qy[..., 1:-1, :-1]

    def coarse(self, f):
        """Nine-point restriction onto the inner half of the next level."""
        w = 0.5 * f[..., :-2, :] + f[..., 1:-1, :] + 0.5 * f[..., 2:, :]
        w = w[..., ::2, :]
        return (0.5 * w[..., :-2] + w[..., 1:-1] + 0.5 * w[..., 2:])[..., ::2]

    def vort2flux(self, gam, levels_q=None):
        """(gamma with its coarse levels filled in, psi per level, (qx, qy) per level)."""
        gam = list(gam)
        nx, ny = self.nx, self.ny
        for l in range(1, self.L):
            g = gam[l].clone()
            g[..., ny // 4:3 * ny // 4 - 1, nx // 4:3 * nx // 4 - 1] = self.coarse(gam[l - 1])
            gam[l] = g
        psi, q = [None] * self.L, [None] * self.L
        for l in range(self.L - 1, -1, -1):
            ring = self.ring(psi[l + 1]) if l < self.L - 1 else None
            psi[l] = self.solve(gam[l] if ring is None else self.edges(gam[l], ring, 1.0), self.lam)
            if levels_q is None or l < levels_q:
                q[l] = self.curl(psi[l], ring)
        return gam, psi, q

    def nonlinear(self, q, uv, gam, ring, hc):
        ax = 0.5 * (q[0][..., 1:, :] + q[0][..., :-1, :]) + uv[0] * hc
        ay = 0.5 * (q[1][..., :, 1:] + q[1][..., :, :-1]) + uv[1] * hc
        g = self.padded(gam, ring)
        fx = torch.zeros_like(q[0])
        fy = torch.zeros_like(q[1])
        m = ay * g[..., :, 1:-1]
        fx[..., :, 1:-1] = 0.5 * (m[..., 1:, :] + m[..., :-1, :])
        m = ax * g[..., 1:-1, :]
        fy[..., 1:-1, :] = -0.5 * (m[..., :, 1:] + m[..., :, :-1])
        return self.rot(fx, fy) / (hc * hc)

    def flat(self, q):
        return torch.cat([q[0].reshape(q[0].shape[:-2] + (-1,)), q[1].reshape(q[1].shape[:-2] + (-1,))], -1)


class PlainRun(Plain):
    """A solve case, step by step."""

    def __init__(self, case, seed):
        super().__init__(case["nx"], case["ny"], case["levels"], case["h"])
        self.case, self.dt, self.re = case, case["dt"], case["re"]
        self.bodies = _bodies(case["bodies"], case["h"])
        self.moving = any(m is not None for _, _, m in self.bodies)
        self.explicit = case["scheme"] == "rkc"
        shape = (self.L, self.ny - 1, self.nx - 1)
        g = torch.from_numpy(_noise(self.nx, self.ny, self.L, self.h, seed)).to(self.dev).reshape(shape)
        self.gam, self.psi, self.q = self.vort2flux(g)
        self.old = [torch.zeros_like(x) for x in self.gam]
        self.hc = [self.h * 2.0 ** l for l in range(self.L)]
        self.implicit = [1.0 + self.lam * self.dt / (2 * self.re * hc * hc) for hc in self.hc]
        self.t, self.cd = 0.0, []
        self.place(0.0)
        if not self.moving:
            self.binv = torch.linalg.inv(self.schur())
        if self.explicit:
            self.coef = _rkc_coefficients(_rkc_stages(case))

    def place(self, t):
        """Body points, their velocities and delta windows at t."""
        xs, vs = [], []
        for xb, _, m in self.bodies:
            if m is None:
                xs.append(xb)
                vs.append(np.zeros_like(xb))
                continue
            r0, v0, th, om = _kinematics(m, t)
            c, s = math.cos(th), math.sin(th)
            xs.append(np.array(r0) + xb @ np.array([[c, -s], [s, c]]).T)
            vs.append(np.array(v0) + om * (xb @ np.array([[-s, -c], [c, -s]]).T))
        self.vel = torch.from_numpy(np.concatenate(vs).T.reshape(-1).copy()).to(self.dev)
        # on the host, where a division is a division: the delta's pieces meet with a step of 1e-9, a
        # point on a grid line sits at such a step, and the distances have to round as written
        x = torch.from_numpy(np.concatenate(xs))
        nx, ny, h = self.nx, self.ny, self.h
        o = torch.tensor([self.case["x0"], self.case["y0"]], dtype=torch.float64)
        cell = torch.floor((x - o) / h).long()
        s = torch.arange(-6, 7)
        i, j = cell[:, 0, None] - 1 + s, cell[:, 1, None] - 1 + s
        gx, gy = h * i.double() + o[0], h * j.double() + o[1]
        rx = [(a - x[:, 0, None]).abs() / h for a in (gx, gx + h / 2)]
        ry = [(a - x[:, 1, None]).abs() / h for a in (gy, gy + h / 2)]
        self.weight = torch.stack([_delta(ry[1])[:, :, None] * _delta(rx[0])[:, None, :],
                                   _delta(ry[0])[:, :, None] * _delta(rx[1])[:, None, :]])
        self.weight = self.weight.reshape(2 * len(x), -1).to(self.dev)
        at = torch.stack([j[:, :, None] * (nx + 1) + i[:, None, :],
                          (nx + 1) * ny + j[:, :, None] * nx + i[:, None, :]])
        self.at = at.reshape(2 * len(x), -1).to(self.dev)

    def gather(self, q, uv=None):
        v = self.flat(q)[..., self.at]
        if uv is not None:
            n = self.at.shape[0] // 2
            v = v + torch.tensor([uv[0]] * n + [uv[1]] * n, dtype=torch.float64, device=self.dev)[:, None] * self.h
        return (v * self.weight).sum(-1)

    def spread(self, f):
        """rot of the forces spread onto the faces."""
        nx, ny = self.nx, self.ny
        q = torch.zeros(f.shape[:-1] + ((nx + 1) * ny + nx * (ny + 1),), dtype=torch.float64, device=self.dev)
        q.index_add_(-1, self.at.reshape(-1), (f[..., None] * self.weight).reshape(f.shape[:-1] + (-1,)))
        nu = (nx + 1) * ny
        return self.rot(q[..., :nu].reshape(f.shape[:-1] + (ny, nx + 1)), q[..., nu:].reshape(f.shape[:-1] + (ny + 1, nx)))

    def schur(self):
        nf = self.at.shape[0]
        step = max(1, min(nf, int(4e7 / (self.nx * self.ny))))
        rows = []
        for c in range(0, nf, step):
            e = torch.eye(nf, dtype=torch.float64, device=self.dev)[c:c + step]
            g = self.spread(e)
            if not self.explicit:
                g = self.solve(g, self.implicit[0])
            z = torch.zeros_like(g)
            rows.append(self.gather(self.vort2flux([g] + [z] * (self.L - 1), 1)[2][0]))
        return torch.cat(rows).T.contiguous()

    def forces(self, q):
        f = self.gather(q, (1.0, 0.0))
        if self.moving:
            f = torch.linalg.solve(self.schur(), f - self.vel * self.h)
        else:
            f = self.binv @ f
        n, k = len(f) // 2, 0
        now = []
        for xb, _, _ in self.bodies:
            part = f.reshape(2, n)[:, k:k + len(xb)].sum(1) * (2 * self.h / self.dt)
            now.append(part)
            k += len(xb)
        self.cd.append(torch.stack(now, 1))
        return f

    def step(self):
        if self.moving:
            self.place(self.t)
        (self.rkc if self.explicit else self.cnab)()
        self.t += self.dt

    def cnab(self):
        gs, bc = [None] * self.L, torch.zeros_like(self.lam)
        for l in range(self.L - 1, -1, -1):
            ring, hc = None, self.hc[l]
            if l < self.L - 1:
                ring = self.ring(self.gam[l + 1])
                bc = self.edges(bc, ring, 0.25 * self.dt / (self.re * hc * hc))
                ring = [0.25 * r for r in ring]
            n = self.nonlinear(self.q[l], (1.0, 0.0), self.gam[l], ring, hc)
            a = self.rot(*self.curl(self.gam[l], None)) * (self.dt / (2 * self.re * hc * hc))
            gs[l] = self.solve(self.gam[l] - a + self.dt * (1.5 * n - 0.5 * self.old[l]) + bc, self.implicit[l])
            self.old[l] = n
        gs, _, q = self.vort2flux(gs, 1)
        f = self.forces(q[0])
        gs[0] = gs[0] - self.solve(self.spread(f), self.implicit[0])
        self.gam, self.psi, self.q = self.vort2flux(gs)

    def rate(self, y, q):
        out = []
        for l in range(self.L):
            ring, hc = None, self.hc[l]
            v = -self.rot(*self.curl(y[l], None))
            if l < self.L - 1:
                ring = self.ring(y[l + 1])
                v = self.edges(v, ring, 1.0)
                ring = [0.25 * r for r in ring]
            out.append(self.nonlinear(q[l], (1.0, 0.0), y[l], ring, hc) + v / (self.re * hc * hc))
        return out

    def rkc(self):
        mu, nu, mt, gt, _ = self.coef
        y0 = self.gam
        f0 = self.rate(y0, self.q)
        y2, y1 = y0, [y + mt[1] * self.dt * f for y, f in zip(y0, f0)]
        for j in range(2, len(mu)):
            y1, _, q = self.vort2flux(y1)
            f = self.rate(y1, q)
            y = [(1 - mu[j] - nu[j]) * a + mu[j] * b + nu[j] * c + self.dt * (mt[j] * d + gt[j] * e)
                 for a, b, c, d, e in zip(y0, y1, y2, f, f0)]
            y2, y1 = y1, y
        y, _, q = self.vort2flux(y1, 1)
        y[0] = y[0] - self.spread(self.forces(q[0]))
        self.gam, self.psi, self.q = self.vort2flux(y)

    def result(self):
        if self.moving:
            for _ in range(MOVING_STEPS):
                self.step()
            self.cd = []
        for _ in range(self.case["steps"]):
            self.step()
        rows = lambda v: torch.stack([x.reshape(-1) for x in v])  # noqa: E731
        out = {"forces": torch.stack(self.cd), "gamma": rows(self.gam)}
        if self.case["precision"] == "fp64":
            out.update(q=torch.stack([self.flat(q) for q in self.q]), psi=rows(self.psi))
            if not self.explicit:
                out["nonlin"] = rows(self.old)
        return out


def exact(case, seed):
    if case["kind"] == "solve":
        return PlainRun(case, seed).result()
    if case["kind"] == "ensemble":
        return [PlainRun(m, seed + k).result() for k, m in enumerate(_members(case))]
    nx, ny = case["nx"], case["ny"]
    f = _fields(case, seed).reshape(-1, ny - 1, nx - 1)
    p = Plain(nx, ny, case.get("levels", 1))
    if case["kind"] == "poisson":
        return p.solve(f, p.lam).reshape(len(f), -1)
    gam, psi, q = p.vort2flux(list(f))
    return [torch.stack([x.reshape(-1) for x in gam]), torch.stack([x.reshape(-1) for x in psi]),
            torch.stack([p.flat(x) for x in q])]
