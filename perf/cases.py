"""What is timed: the calls that programs built on this framework make, over the sizes they use.

A case is a dict of plain values; ``kind`` names the call:

  transform  Chebyshev.forward_fft and backward_fft of a field along one axis
  field      Field.dealias.backward / forward: 2-D transforms onto and back from the 3/2 grid
  adi        solverplan_hholtz2d_adi: right-hand side, old term and solve of one implicit step
  exact      solverplan_hholtz2d_fd: the same with the unsplit operator (two dense products)
  update     NavierStokes.update(): one step per call, as a script's own loop makes it
  iterate    NavierStokes.iterate(): the library's time loop, several steps a call
  batch      FusedBatch.step() of instances of different shapes and Rayleigh numbers, tuned and captured
  batch_host FusedBatch.step_host(): the same with the fields in pinned host memory on both sides
  horizon    HorizonGradient.value_and_grad(): objective and gradient over a horizon of steps
  autograd   update() of fields that need gradients, and torch.autograd back through it

``exact`` restates each of them with dense matrices in torch on the CPU, in 64 bits.
"""
import math

import numpy as np
import torch

import pypde_gb300 as pg
from pypde_gb300.navier.fused import FusedBatch
from pypde_gb300.navier.fused_adjoint import FusedAdjoint, HorizonGradient
from pypde_gb300.navier.rbc2d import NavierStokes

F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the shortest call: a small field transformed there and back (scripts, diagnostics; the tests'
        # and the benchmark's smallest size): all latency
        {"name": "transform_33", "kind": "transform", "n": 33, "lines": 33},
        # the longest lines of the benchmark's transform sizes
        {"name": "transform_1025", "kind": "transform", "n": 1025, "lines": 1025},
        # the 2-D transforms of a mid-sized field onto the 3/2 grid and back, as convection terms take them
        {"name": "field_193x129", "kind": "field", "nx": 193, "ny": 129, "side": "CD"},
        # one implicit diffusion step with the split operator, at the benchmark's size
        {"name": "adi_257", "kind": "adi", "nx": 257, "ny": 257, "lam": 0.01},
        # the unsplit solve: dense products with the eigenvectors along one axis
        {"name": "exact_513", "kind": "exact", "nx": 513, "ny": 513, "lam": 0.01},
        # a script's own loop on the reference's default configuration (50 x 50, sidewalls insulated:
        # lengths that no FFT of factors 2 and 3 divides)
        {"name": "update_50", "kind": "update", "case": "rbc", "nx": 50, "ny": 50, "ra": 5e3, "dt": 0.2,
         "aspect": 1.0, "dealias": True, "integrator": "eu", "beta": 1.0},
        # the library's time loop on the smallest of the benchmark's flows
        {"name": "iterate_65", "kind": "iterate", "case": "linear", "nx": 65, "ny": 65, "ra": 1e5, "dt": 0.01,
         "aspect": 1.0, "dealias": True, "integrator": "eu", "beta": 1.0, "steps": 10},
        # ... and on the largest
        {"name": "iterate_513x257", "kind": "iterate", "case": "linear", "nx": 513, "ny": 257, "ra": 1e8, "dt": 1e-3,
         "aspect": 2.0, "dealias": True, "integrator": "eu", "beta": 1.0, "steps": 2},
        # many flows at once (parameter studies): shapes of {33, 65, 129} per axis, Ra 1e4 .. 1e7
        {"name": "batch_64", "kind": "batch", "count": 64, "sizes": "33,65,129", "dt": 0.005},
        # the same fed from and read back to the host every step
        {"name": "batch_host_64", "kind": "batch_host", "count": 64, "sizes": "33,65,129", "dt": 0.005},
        # the gradient of a steady-state search: forward horizon, checkpoints, reverse sweep
        {"name": "horizon_129", "kind": "horizon", "nx": 129, "ny": 129, "ra": 1e5, "dt": 0.01, "steps": 60,
         "every": 20},
        # a step inside a torch program that differentiates it
        {"name": "autograd_65x49", "kind": "autograd", "nx": 65, "ny": 49, "ra": 1e5, "dt": 0.01},
    ]


# sizes whose transforms (of N and of int(1.5 N) points) are FFTs of factors 2 and 3, as users pick
# them, beside arbitrary ones
_SMOOTH = (17, 25, 33, 49, 65, 73, 97, 129, 145, 163, 193, 257, 289, 385, 433, 513)


def _size(rng, lo, hi, smooth=0.5):
    if rng.random() < smooth:
        return rng.choice([n for n in _SMOOTH if lo <= n <= hi])
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _flow(rng, kind, lo, hi):
    return {"kind": kind, "case": rng.choice(["linear", "rbc", "zero"]), "nx": _size(rng, lo, hi),
            "ny": _size(rng, lo, hi), "ra": round(10 ** rng.uniform(4, 8), 1), "dt": rng.choice([1e-3, 2e-3, 5e-3, 0.01]),
            "aspect": rng.choice([1.0, 2.0]), "dealias": rng.random() < 0.8,
            "integrator": rng.choice(["eu", "eu", "rk3"]), "beta": rng.choice([1.0, 1.0, 0.5])}


def draw(rng):
    kind = rng.choice(["transform", "transform", "field", "field", "adi", "exact", "update", "iterate", "batch",
                       "batch_host", "horizon", "autograd"])
    if kind == "transform":
        n = rng.choice([_size(rng, 17, 513), 769, 1025]) if rng.random() < 0.6 else _size(rng, 17, 400, smooth=0.0)
        return {"kind": kind, "n": n, "lines": int(round(math.exp(rng.uniform(math.log(17), math.log(1025)))))}
    if kind == "field":
        return {"kind": kind, "nx": _size(rng, 17, 513), "ny": _size(rng, 17, 513), "side": rng.choice(["CD", "CN"])}
    if kind in ("adi", "exact"):
        hi = 1025 if kind == "adi" else 513
        return {"kind": kind, "nx": _size(rng, 17, hi, smooth=0.3), "ny": _size(rng, 17, hi, smooth=0.3),
                "lam": round(10 ** rng.uniform(-4, -1), 6)}
    if kind == "update":
        return _flow(rng, kind, 17, 193)
    if kind == "iterate":
        c = _flow(rng, kind, 25, 289)
        c["steps"] = rng.randint(2, 10)
        return c
    if kind in ("batch", "batch_host"):
        return {"kind": kind, "count": rng.randint(6, 40), "dt": rng.choice([1e-3, 2e-3, 5e-3]),
                "sizes": ",".join(str(n) for n in sorted(rng.sample(
                    [17, 25, 33, 41, 49, 65, 73, 81, 97, 113, 129], rng.randint(2, 4))))}
    if kind == "horizon":
        return {"kind": kind, "nx": _size(rng, 25, 129), "ny": _size(rng, 25, 129), "dt": 0.005,
                "ra": round(10 ** rng.uniform(4, 6), 1), "steps": rng.randint(20, 60), "every": rng.choice([10, 20])}
    return {"kind": kind, "nx": _size(rng, 25, 129), "ny": _size(rng, 25, 129), "dt": 0.005,
            "ra": round(10 ** rng.uniform(4, 6), 1)}


# ------------------------------------------------------------------ inputs
def _spectrum(rng, shape, amp):
    """Coefficients of a resolved field: random, falling to about 1e-5 of the largest at the highest modes."""
    i, j = np.arange(shape[0])[:, None], np.arange(shape[1])[None, :]
    return amp * rng.standard_normal(shape) * np.exp(-8.0 * i / shape[0] - 8.0 * j / shape[1])


def _fields(seed, nx, ny, index=0):
    """Velocity, temperature deviation and pressure coefficients of a developed flow."""
    rng = np.random.default_rng([seed, index])
    inner = (nx - 2, ny - 2)
    return {"U": _spectrum(rng, inner, 0.05), "V": _spectrum(rng, inner, 0.05), "T": _spectrum(rng, inner, 0.05),
            "pres": _spectrum(rng, (nx, ny), 0.02)}


def _instances(case, seed):
    """(nx, ny, Ra) of a batch: shapes from the case's sizes, Ra over three decades.  Which shapes a
    batch has belongs to the case, not to the seed."""
    sizes = [int(s) for s in case["sizes"].split(",")]
    rng = np.random.default_rng(99)
    shapes = rng.choice(sizes, size=(case["count"], 2))
    ra = 10.0 ** rng.uniform(4, 7, case["count"])
    return [(int(nx), int(ny), float(r)) for (nx, ny), r in zip(shapes, ra)]


def _solver(nx, ny, ra, dt, case="linear", aspect=1.0, dealias=True, integrator="eu", beta=1.0):
    return NavierStokes(case=case, shape=(nx, ny), ra=ra, pr=1.0, dt=dt, aspect=aspect, dealias=dealias,
                        integrator=integrator, beta=beta, tsave=None)


def _flow_options(case):
    return {k: case[k] for k in ("case", "aspect", "dealias", "integrator", "beta") if k in case}


def _seeded(ns, fields):
    for k, v in fields.items():
        getattr(ns, k).vhat = v
    return ns


def _uniform(seed, *shape):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, shape)


def _device(x):
    return torch.as_tensor(x, dtype=F64, device="cuda")


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "transform":
        s["base"] = pg.Base(case["n"], "CH")
        s["v"] = _device(_uniform(seed, case["n"], case["lines"]))
    elif kind == "field":
        s["field"] = pg.Field([pg.Base(case["nx"], case["side"], dealias=3 / 2), pg.Base(case["ny"], "CD", dealias=3 / 2)])
        s["vhat"] = _device(_spectrum(np.random.default_rng(seed), (case["nx"] - 2, case["ny"] - 2), 0.1))
    elif kind in ("adi", "exact"):
        make = pg.solverplan_hholtz2d_adi if kind == "adi" else pg.solverplan_hholtz2d_fd
        s["plan"] = make(pg.Field([pg.Base(case["nx"], "CD"), pg.Base(case["ny"], "CD")]).xs, lam=case["lam"])
        s["f"] = _device(_uniform(seed, case["nx"], case["ny"]))
        s["old"] = _device(_spectrum(np.random.default_rng([seed, 1]), (case["nx"] - 2, case["ny"] - 2), 0.1))
    elif kind in ("update", "iterate"):
        ns = _solver(case["nx"], case["ny"], case["ra"], case["dt"], **_flow_options(case))
        _seeded(ns, _fields(seed, case["nx"], case["ny"]))
        s["ns"], s["time"] = ns, case.get("steps", 1) * case["dt"]
        s["x0"] = ns.fused().state_arena.clone()
        if kind == "iterate":
            ns.fused().capture(1)
    elif kind in ("batch", "batch_host"):
        solvers = [_seeded(_solver(nx, ny, ra, case["dt"]), _fields(seed, nx, ny, k))
                   for k, (nx, ny, ra) in enumerate(_instances(case, seed))]
        fb = s["fb"] = FusedBatch(solvers)
        fb.autotune(reps=2)
        s["x0"] = fb.state_arena.clone()
        if kind == "batch":
            fb.capture(1, groups="shape")
        else:
            fb.host_pipeline()
            s["x0"] = s["x0"].cpu()
            s["host"] = torch.empty_like(s["x0"]).pin_memory()
    elif kind == "horizon":
        ns = _seeded(_solver(case["nx"], case["ny"], case["ra"], case["dt"]), _fields(seed, case["nx"], case["ny"]))
        fa = FusedAdjoint([ns])
        s["x"] = fa.state_arena.clone()
        s["hg"] = HorizonGradient(fa, case["steps"], case["every"])
        s["hg"].value_and_grad(s["x"])
    else:
        s["ns"] = _solver(case["nx"], case["ny"], case["ra"], case["dt"])
        f = _fields(seed, case["nx"], case["ny"])
        s["x"] = {k: _device(v) for k, v in f.items()}
        s["w"] = {k: _device(_uniform([seed, i], *v.shape)) for i, (k, v) in enumerate(f.items())}
    return s


def run(s):
    kind = s["kind"]
    if kind == "transform":
        c = s["base"].forward_fft(s["v"])
        return {"coefficients": c, "values": s["base"].backward_fft(c)}
    if kind == "field":
        v = s["field"].dealias.backward(s["vhat"])
        return {"values": v, "coefficients": s["field"].dealias.forward(v)}
    if kind in ("adi", "exact"):
        plan = s["plan"]
        return plan.solve_lhs(plan.solve_rhs(s["f"]) + plan.solve_old(s["old"]))
    if kind in ("update", "iterate"):
        ns = s["ns"]
        ns.fused().state_arena.copy_(s["x0"])
        if kind == "update":
            ns.update()
        else:
            ns.reset_time()
            ns.iterate(s["time"])
        return {k: getattr(ns, k).vhat for k in ("U", "V", "T", "P", "pres")}
    if kind == "batch":
        s["fb"].state_arena.copy_(s["x0"])
        s["fb"].step()
        return s["fb"].state_arena
    if kind == "batch_host":
        s["host"].copy_(s["x0"])
        s["fb"].step_host(s["host"], wait=True)
        torch.cuda.current_stream().synchronize()  # the fields are read on the host
        return s["host"]
    if kind == "horizon":
        J, g = s["hg"].value_and_grad(s["x"])
        return {"J": J, "gradient": g}
    ns = s["ns"]
    x = {k: v.detach().requires_grad_(True) for k, v in s["x"].items()}
    for k, v in x.items():
        getattr(ns, k).vhat = v
    ns.update()
    y = {k: getattr(ns, k).vhat for k in x}
    g = torch.autograd.grad(list(y.values()), list(x.values()), [s["w"][k] for k in y])
    return {"state": [v.detach() for v in y.values()], "gradient": list(g)}


# ------------------------------------------------------------------ work
def _dct_flops(n):
    return 2.5 * n * math.log2(max(2.0, 2.0 * (n - 1)))


def _step_work(nx, ny, dealias=True, stages=1):
    """One step of one flow: 20 transforms a grid line pair, two dense products, about 150 flops a
    mode in stencils, recurrences and banded sweeps; the state read and written, the tables read."""
    nd, md = (int(1.5 * nx), int(1.5 * ny)) if dealias else (nx, ny)
    fl = (6 * (ny - 2) + 3 * ny) * _dct_flops(nd) + 11 * nd * _dct_flops(md)
    fl += 4.0 * (nx - 2) * (ny - 2) * ny + 150.0 * nx * ny
    by = 8.0 * (2 * 5 * nx * ny + 2 * ny * ny + 4 * nx * ny)
    return {"flops": stages * fl, "bytes": by}


def work(case):
    kind = case["kind"]
    if kind == "transform":
        return {"flops": 2 * case["lines"] * _dct_flops(case["n"]), "bytes": 3 * 8.0 * case["n"] * case["lines"]}
    nx, ny = case.get("nx"), case.get("ny")
    if kind == "field":
        nd, md = int(1.5 * nx), int(1.5 * ny)
        return {"flops": (ny + ny) * _dct_flops(nd) + 2 * nd * _dct_flops(md), "bytes": 8.0 * (2 * nx * ny + nd * md)}
    if kind in ("adi", "exact"):
        dense = 0.0 if kind == "adi" else 6.0 * nx * ny * ny
        return {"flops": 30.0 * nx * ny + dense, "bytes": 8.0 * (3 * nx * ny + (0 if kind == "adi" else 3 * ny * ny + 4 * nx * ny))}
    if kind in ("update", "iterate"):
        w = _step_work(nx, ny, case["dealias"], 3 if case["integrator"] == "rk3" else 1)
        return {"flops": case.get("steps", 1) * w["flops"], "bytes": w["bytes"]}
    if kind in ("batch", "batch_host"):
        each = [_step_work(a, b) for a, b, _ in _instances(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("flops", "bytes")}
    w = _step_work(nx, ny)
    if kind == "horizon":  # forward and reverse sweep; a reverse step is about two forward ones
        return {"flops": 3 * case["steps"] * w["flops"], "bytes": w["bytes"]}
    return {"flops": 3 * w["flops"], "bytes": 2 * w["bytes"]}


# ------------------------------------------------------------------ 64 bits on the CPU
def _cos(n):
    """T_k(x_j) on the ascending Gauss-Lobatto points x_j = -cos(pi j / (n - 1))."""
    j, k = np.arange(n)[:, None], np.arange(n)[None, :]
    return np.where(k % 2, -1.0, 1.0) * np.cos(np.pi * ((j * k) % (2 * (n - 1))) / (n - 1))


def _to_values(n):
    return torch.from_numpy(_cos(n))


def _to_coefficients(n):
    w = np.full(n, 1.0)
    w[0] = w[-1] = 0.5
    return torch.from_numpy(2.0 / (n - 1) * w[:, None] * _cos(n).T * w[None, :])


def _stencil(key, n):
    if key == "CH":
        return torch.eye(n, dtype=F64)
    S = np.zeros((n, n - 2))
    k = np.arange(n - 2)
    S[k, k] = 1.0
    S[k + 2, k] = -1.0 if key == "CD" else -((k / (k + 2.0)) ** 2)
    return torch.from_numpy(S)


def _derivative(n):
    D = np.zeros((n, n))
    for j in range(n):
        D[j, j + 1::2] = 2.0 * np.arange(j + 1, n, 2)
    D[0] *= 0.5
    return torch.from_numpy(D)


def _pinv(n):
    """Rows 2.. of the banded pseudo-inverse of the second derivative, with pypde's cut-offs."""
    B = np.zeros((n, n))
    i = np.arange(2, n - 2)
    B[i, i] = -1.0 / (2.0 * (i * i - 1.0))
    i = np.arange(2, n - 4)
    B[i, i + 2] = 1.0 / (4.0 * i * (i + 1.0))
    i = np.arange(2, n)
    B[i, i - 2] = 1.0 / (4.0 * i * (i - 1.0))
    B[2, 0] *= 2.0
    B[np.abs(B) < 1e-12] = 0.0
    return torch.from_numpy(B[2:])


def _inverse_stencil(key, n):
    S = _stencil(key, n)
    return torch.linalg.solve(S.T @ S, S.T.contiguous())


class _Adi:
    def __init__(self, keys, shape, lam, scale=(1.0, 1.0)):
        self.B, self.BS, self.lu = [], [], []
        for key, n, s in zip(keys, shape, scale):
            S, B = _stencil(key, n), _pinv(n)
            self.B.append(B)
            self.BS.append(B @ S)
            self.lu.append(torch.linalg.lu_factor(B @ S - lam / s ** 2 * S[2:]))

    def __call__(self, rhs, old):
        b = self.B[0] @ rhs @ self.B[1].T + self.BS[0] @ old @ self.BS[1].T
        b = torch.linalg.lu_solve(*self.lu[0], b)
        return torch.linalg.lu_solve(*self.lu[1], b.T.contiguous()).T


class _FastDiagonal:
    """(A_x + alpha_i C_x) per eigenvalue i of the y operator; ``lam``: the Helmholtz form."""

    def __init__(self, key, shape, scale=(1.0, 1.0), lam=None):
        (nx, ny), (sx, sy) = shape, scale
        Sx, Sy, self.Bx, By = _stencil(key, nx), _stencil(key, ny), _pinv(nx), _pinv(ny)
        A, C = Sx[2:] / sx ** 2, self.Bx @ Sx
        Cy = By @ Sy
        Ci = np.linalg.inv(Cy.numpy())
        w, Q = np.linalg.eig(Ci @ (Sy[2:] * (1.0 / sy ** 2)).numpy())
        w, Q = np.real(w), np.real(Q)
        order = np.argsort(w)[::-1]
        w, Q = w[order].copy(), np.ascontiguousarray(Q[:, order])
        Qi = np.linalg.inv(Q)
        self.Q, self.H, self.Qi, self.C = (torch.from_numpy(np.ascontiguousarray(m)) for m in (Q, Qi @ Ci @ By.numpy(), Qi, C.numpy()))
        w = torch.from_numpy(w)
        alpha = w if lam is None else 1.0 - lam * w
        A = A if lam is None else -lam * A
        M = A[None] + alpha[:, None, None] * C[None]
        if lam is None:  # the constant mode: rows 1.., first unknown zero
            for i in torch.nonzero(alpha.abs() < 1e-10).flatten().tolist():
                M[i, 0, :] = 0.0
                M[i, :, 0] = 0.0
                M[i, 0, 0] = 1e300
        self.lu = torch.linalg.lu_factor(M)

    def solve(self, b):
        x = torch.linalg.lu_solve(*self.lu, b.T.contiguous()[:, :, None])[:, :, 0].T
        return x @ self.Q.T

    def __call__(self, rhs, old=None):
        b = self.Bx @ rhs @ self.H.T
        if old is not None:
            b = b + self.C @ old @ self.Qi.T
        return self.solve(b)


class _Step:
    """One time step of the flow with dense operators (differentiable by torch)."""

    def __init__(self, nx, ny, ra, dt, case="linear", aspect=1.0, dealias=True, integrator="eu", beta=1.0):
        self.dt, self.beta = dt, beta
        self.nu = self.kappa = math.sqrt(1.0 / ra)
        self.scale = sx, sz = aspect * 0.5, 0.5
        tk = "CN" if case == "rbc" else "CD"
        self.shape, self.grid = (nx, ny), (int(1.5 * nx), int(1.5 * ny)) if dealias else (nx, ny)
        if integrator == "rk3":
            self.stages = list(zip((8 / 15, 2 / 15, 1 / 3), (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)))
        else:
            self.stages = [(1.0, 1.0, 0.0)]
        self.S = {F: (_stencil(k, nx), _stencil("CD", ny)) for F, k in (("U", "CD"), ("V", "CD"), ("T", tk))}
        self.S["P"] = (_stencil("CN", nx), _stencil("CN", ny))
        self.D = (_derivative(nx) / sx, _derivative(ny) / sz)
        self.back = [_to_values(g)[:, :n] for g, n in zip(self.grid, self.shape)]
        self.forw = [_to_coefficients(g)[:n] for g, n in zip(self.grid, self.shape)]
        self.inv = (_inverse_stencil("CD", nx), _inverse_stencil("CD", ny))
        self.adi = [{F: _Adi((tk if F == "T" else "CD", "CD"), self.shape,
                             dt * a * beta * (self.kappa if F == "T" else self.nu), self.scale) for F in "UT"}
                    for a, _, _ in self.stages]
        self.poisson = _FastDiagonal("CN", self.shape, self.scale)
        self._lift(case, tk)

    def _lift(self, case, tk):
        nx, ny = self.shape
        if case == "zero":
            y = -np.cos(np.pi * np.arange(ny) / (ny - 1)) * self.scale[1]
            x = y * 2.0 / (y[-1] - y[0])
            with np.errstate(divide="ignore", invalid="ignore"):
                prof = np.where(x < 0, -0.02 * x / (0.02 + x + 1) * 0.5, 0.02 * x / (0.02 - x + 1) * -0.5)
            two = torch.from_numpy(np.stack([prof, prof]))
            c = _to_coefficients(ny) @ two.T      # the profile along y, the same at both sidewalls
            lift = torch.zeros((nx, ny), dtype=F64)
            lift[0], lift[1] = 0.5 * (c[:, 0] + c[:, 1]), 0.5 * (c[:, 1] - c[:, 0])
        else:                                    # 1/2 at the bottom, -1/2 at the top
            lift = torch.zeros((nx, ny), dtype=F64)
            lift[0, 1] = -0.5
        self.lift = lift
        self.dlift = self.back[0] @ (lift @ self.D[1].T) @ self.back[1].T
        self.ddlift = lift @ (self.D[1] @ self.D[1]).T

    def cheb(self, F, c):
        return self.S[F][0] @ c @ self.S[F][1].T

    def values(self, c):
        return self.back[0] @ c @ self.back[1].T

    def grad(self, c):
        return self.D[0] @ c, c @ self.D[1].T

    def __call__(self, X):
        U, V, T, pres = (X[k] for k in ("U", "V", "T", "pres"))
        dt, old = self.dt, None
        for (a, b, c), adi in zip(self.stages, self.adi):
            Tc = self.cheb("T", T) + self.lift
            ux, uz = self.values(self.cheb("U", U)), self.values(self.cheb("V", V))
            wx, wz = (ux, uz) if old is None else (b * ux + c * old[0], b * uz + c * old[1])
            if old is None:
                wx, wz = b * wx, b * wz
            px, pz = self.grad(pres)
            rhs = {}
            for F, f in (("U", U), ("V", V), ("T", T)):
                dx, dz = self.grad(self.cheb(F, f))
                n = wx * self.values(dx) + wz * self.values(dz)
                if F == "T":
                    n = n + wz * self.dlift
                r = -dt * (self.forw[0] @ n @ self.forw[1].T)
                if self.beta != 1.0:
                    e = dt * a * (1.0 - self.beta) * (self.kappa if F == "T" else self.nu)
                    r = r + e * (self.D[0] @ dx + dz @ self.D[1].T)
                rhs[F] = r
            rhs["U"] = rhs["U"] - dt * a * px
            rhs["V"] = rhs["V"] - dt * a * pz + dt * a * Tc
            rhs["T"] = rhs["T"] + dt * a * self.kappa * self.ddlift
            U, V, T = adi["U"](rhs["U"], U), adi["U"](rhs["V"], V), adi["T"](rhs["T"], T)
            div = self.D[0] @ self.cheb("U", U) + self.cheb("V", V) @ self.D[1].T
            P = self.poisson(div)
            mask = torch.ones_like(P)
            mask[0, 0] = 0.0
            P = P * mask
            Pc = self.cheb("P", P)
            pres = pres - self.nu * self.beta * div + Pc / (dt * a)
            gx, gz = self.grad(Pc)
            U = U - self.inv[0] @ gx @ self.inv[1].T
            V = V - self.inv[0] @ gz @ self.inv[1].T
            old = (ux, uz)
        return {"U": U, "V": V, "T": T, "P": P, "pres": pres}


def _cpu(fields):
    return {k: torch.from_numpy(v) for k, v in fields.items()}


def exact(case, seed):
    kind, nx, ny = case["kind"], case.get("nx"), case.get("ny")
    if kind == "transform":
        c = _to_coefficients(case["n"]) @ torch.from_numpy(_uniform(seed, case["n"], case["lines"]))
        return {"coefficients": c, "values": _to_values(case["n"]) @ c}
    if kind == "field":
        nd, md = int(1.5 * nx), int(1.5 * ny)
        c = torch.from_numpy(_spectrum(np.random.default_rng(seed), (nx - 2, ny - 2), 0.1))
        v = _to_values(nd)[:, :nx] @ _stencil(case["side"], nx) @ c @ (_to_values(md)[:, :ny] @ _stencil("CD", ny)).T
        back = [_inverse_stencil(k, int(1.5 * n)) @ _to_coefficients(int(1.5 * n)) for k, n in ((case["side"], nx), ("CD", ny))]
        return {"values": v, "coefficients": (back[0][:nx - 2] @ v @ back[1][:ny - 2].T)}
    if kind in ("adi", "exact"):
        f = torch.from_numpy(_uniform(seed, nx, ny))
        old = torch.from_numpy(_spectrum(np.random.default_rng([seed, 1]), (nx - 2, ny - 2), 0.1))
        if kind == "adi":
            return _Adi(("CD", "CD"), (nx, ny), case["lam"])(f, old)
        return _FastDiagonal("CD", (nx, ny), lam=case["lam"])(f, old)
    if kind in ("update", "iterate"):
        step = _Step(nx, ny, case["ra"], case["dt"], **_flow_options(case))
        X = _cpu(_fields(seed, nx, ny))
        for _ in range(case.get("steps", 1)):
            X = step(X)
        return {k: X[k] for k in ("U", "V", "T", "P", "pres")}
    if kind in ("batch", "batch_host"):  # the arena: flow after flow, ordered by shape
        flows = _instances(case, seed)
        out = []
        for k in sorted(range(len(flows)), key=lambda k: flows[k][:2]):
            a, b, ra = flows[k]
            X = _Step(a, b, ra, case["dt"])(_cpu(_fields(seed, a, b, k)))
            out += [X[f].reshape(-1) for f in ("U", "V", "T", "P", "pres")]
        return torch.cat(out)
    step = _Step(nx, ny, case["ra"], case["dt"])
    if kind == "horizon":
        if case["steps"] * nx * ny * (nx + ny) > 4e8:
            return None
        x = {k: v.requires_grad_(True) for k, v in _cpu(_fields(seed, nx, ny)).items() if k != "pres"}
        X = {**x, "pres": torch.zeros((nx, ny), dtype=F64)}
        for _ in range(case["steps"]):
            X = step(X)
        J = torch.sqrt(sum(((X[k] - x[k]) ** 2).sum() for k in x))
        g = torch.autograd.grad(J, [x["U"], x["V"], x["T"]])
        rest = torch.zeros((nx - 2) * (ny - 2) + nx * ny, dtype=F64)
        return {"J": J.detach().reshape(1), "gradient": torch.cat([v.reshape(-1) for v in g] + [rest])}
    x = {k: v.requires_grad_(True) for k, v in _cpu(_fields(seed, nx, ny)).items()}
    X = step(x)
    w = [torch.from_numpy(_uniform([seed, i], *x[k].shape)) for i, k in enumerate(x)]
    g = torch.autograd.grad([X[k] for k in x], list(x.values()), w)
    return {"state": [X[k].detach() for k in x], "gradient": list(g)}
