"""Performance cases of the step engine: what a user has it do, through the
solvers and plans a user calls.

A case is one pass of one of four calls:

* ``step``  - ``SpectralSolver*.step(U, dt)``: one step of a host-driven loop;
* ``run``   - ``SpectralSolver*.run(U0, 0, t_end)``: a whole CFL-driven solve;
* ``fixed`` - ``Plan.run_``: a block of fixed steps on a resident state;
* ``cfl``   - ``Plan.run_cfl_``: a chunk of device-controlled CFL steps on a
  batch of solves (the form ensembles and the serving loop issue).

``exact`` restates the same pass in float64 with torch and numpy alone: full
N-D complex transforms for the Fourier grids, dense differentiation matrices
for the Legendre grids.
"""
from __future__ import annotations

import math
from typing import Any, Dict, List, Tuple

import numpy as np
import torch

TWO_PI = 2.0 * math.pi
FILTER = {"enabled": True, "p": 8, "alpha": 36.0}


def _case(name: str, kind: str, call: str, nx: int, ny: int = 0, nz: int = 0, *, batch: int = 1, steps: int = 1,
          filt: bool = True, precision: str = "fp32", scheme: str = "rk4") -> Dict[str, Any]:
    c = dict(kind=kind, call=call, nx=nx, ny=ny, nz=nz, batch=batch, steps=steps, filter=filt, precision=precision,
             scheme=scheme)
    return dict(c, name=name) if name else c


def listed() -> List[Dict[str, Any]]:
    return [
        # the smallest call: one step of a 1D shock tube in a user's own loop
        _case("sod1d 256 step", "euler", "step", 256),
        # a served group of 1D shock tubes: 64 resident solves, a chunk of CFL steps
        _case("sod1d 1024 x64 cfl", "euler", "cfl", 1024, batch=64, steps=16),
        # an ordinary 2D shear-layer step in a user's own loop
        _case("khi2d 128 step", "euler", "step", 128, 128),
        # the whole public solve: CFL loop with time-step control and records
        _case("khi2d 256 run", "euler", "run", 256, 256, steps=8),
        # the largest size group of the shear-layer ensemble: 16 solves, a chunk of CFL steps
        _case("khi2d 512 x16 cfl", "euler", "cfl", 512, 512, batch=16, steps=3, filt=False),
        # the largest shipped 2D grid; axes of 2^8 3 5 and 2^4 3^3 5 points
        _case("khi2d 3840x2160 step", "euler", "step", 3840, 2160),
        # the usual 3D size, filter on
        _case("tgv3d 64 step", "euler", "step", 64, 64, 64),
        # the largest single solve: the 3D vortex benchmark, mask-only filter, fixed steps
        _case("tgv3d 256 fixed", "euler", "fixed", 256, 256, 256, steps=2, filt=False),
        # 2D MHD with the projection after every stage
        _case("ot2d 512 step", "mhd", "step", 512, 512),
        # 3D MHD with the projection after every stage
        _case("alfven3d 128 step", "mhd", "step", 128, 128, 128),
        # collocation with walls, tensor-core contractions
        _case("lgl2d 513 bf16x3 step", "lgl", "step", 513, 513, filt=False, precision="bf16x3"),
        # collocation with walls at the grid's default precision, nodal filter on
        _case("lgl2d 257 fp32 step", "lgl", "step", 257, 257),
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2(rng, lo: int, hi: int) -> int:
    a, b = int(math.log2(lo)), int(math.log2(hi))
    return 1 << rng.randint(a, b)


def _smooth(rng, lo: int, hi: int) -> int:
    """A Fourier axis length: a power of two half of the time, else any 2^a 3^b 5^c
    (odd ones among them)."""
    if rng.random() < 0.5:
        return _pow2(rng, lo, hi)
    target = _log_int(rng, lo, hi)
    best = lo
    for a in range(13):
        for b in range(8):
            for c in range(6):
                n = 2 ** a * 3 ** b * 5 ** c
                if lo <= n <= hi and abs(n - target) < abs(best - target):
                    best = n
    return best


def draw(rng) -> Dict[str, Any]:
    family = rng.choice(["sod", "khi", "khi", "khi batch", "tgv", "tgv", "ot", "alfven", "lgl", "lgl"])
    filt = rng.random() < 0.6
    scheme = "rk2" if rng.random() < 0.15 else "rk4"
    if family == "sod":
        n = _smooth(rng, 64, 4096)
        if rng.random() < 0.5:
            return _case("", "euler", "step", n, filt=filt, scheme=scheme)
        return _case("", "euler", "cfl", n, batch=_log_int(rng, 2, 200), steps=rng.randint(4, 16), filt=filt,
                     scheme=scheme)
    if family == "khi":
        call = rng.choice(["step", "fixed", "run"])
        return _case("", "euler", call, _smooth(rng, 32, 1024), _smooth(rng, 32, 1024),
                     steps=1 if call == "step" else rng.randint(2, 8), filt=filt, scheme=scheme)
    if family == "khi batch":
        n = rng.choice([64, 128, 256, 512])
        return _case("", "euler", "cfl", n, n, batch=max(2, _log_int(rng, 2, 128) * 64 // n), steps=rng.randint(2, 4),
                     filt=filt, scheme=scheme)
    if family == "tgv":
        n = [_smooth(rng, 16, 200) for _ in range(3)]
        return _case("", "euler", rng.choice(["step", "fixed"]), *n, steps=1, filt=filt, scheme=scheme)
    if family == "ot":
        return _case("", "mhd", "step", _pow2(rng, 32, 512), _pow2(rng, 32, 512), filt=filt, scheme=scheme)
    if family == "alfven":
        return _case("", "mhd", "step", *[_pow2(rng, 16, 128) for _ in range(3)], filt=filt, scheme=scheme)
    precision = rng.choice(["fp32", "bf16x3", "fp64"])
    hi = 513 if precision == "bf16x3" else 321 if precision == "fp32" else 161
    return _case("", "lgl", "step", _log_int(rng, 17, hi), _log_int(rng, 17, hi), filt=filt, precision=precision,
                 scheme=scheme)


# ------------------------------------------------------------------ inputs
def _ndim(c) -> int:
    return 3 if c["nz"] else 2 if c["ny"] else 1


def _shape(c) -> Tuple[int, ...]:
    return tuple(n for n in (c["nz"], c["ny"], c["nx"]) if n)


def _gamma(c) -> float:
    return 5.0 / 3.0 if c["kind"] == "mhd" else 1.4


def _ncomp(c) -> int:
    return 8 if c["kind"] == "mhd" else _ndim(c) + 2


def _cfl(c) -> float:
    return {1: 0.4, 2: 0.3, 3: 0.25}[_ndim(c)]


def _lengths(c) -> Tuple[float, ...]:
    d = _ndim(c)
    if c["kind"] == "lgl":
        return (2.0, 2.0)
    if c["kind"] == "mhd":
        return (TWO_PI, TWO_PI) if d == 2 else (1.0, 1.0, 1.0)
    return {1: (1.0,), 2: (1.0, 1.0), 3: (TWO_PI,) * 3}[d]


def _device() -> torch.device:
    return torch.device("cuda", torch.cuda.current_device())


def _axis(n: int, length: float) -> torch.Tensor:
    return torch.arange(n, dtype=torch.float64, device=_device()) * (length / n)


def _conservative(rho, vel, p, gamma):
    vel = [v.expand_as(rho) for v in vel]
    E = p / (gamma - 1.0) + 0.5 * rho * sum(v * v for v in vel)
    return torch.stack([rho] + [rho * v for v in vel] + [E.expand_as(rho)])


def _sod(c, r) -> torch.Tensor:
    """Periodic smoothed shock tube; edges and states drawn per solve."""
    x = _axis(c["nx"], 1.0)
    w = max(0.005, 2.5 / c["nx"])
    a, b = r.uniform(0.2, 0.3), r.uniform(0.7, 0.8)
    s = 0.5 * (torch.tanh((x - a) / w) - torch.tanh((x - b) / w))
    rl, pl = r.uniform(0.12, 0.3), r.uniform(0.1, 0.3)
    return _conservative(rl + (1.0 - rl) * s, [torch.zeros_like(x)], pl + (1.0 - pl) * s, 1.4)


def _khi(c, r) -> torch.Tensor:
    """Double shear layer on the unit square with a drawn multi-mode perturbation."""
    x, y = _axis(c["nx"], 1.0)[None, :], _axis(c["ny"], 1.0)[:, None]
    s = torch.tanh((y - 0.25) / 0.05) - torch.tanh((y - 0.75) / 0.05) - 1.0
    g = torch.exp(-(y - 0.25) ** 2 / 0.0025) + torch.exp(-(y - 0.75) ** 2 / 0.0025)
    v = sum(r.uniform(0.002, 0.01) * torch.sin(TWO_PI * m * x + r.uniform(0.0, TWO_PI)) for m in (1, 2, 3)) * g
    rho = (1.5 + 0.5 * s).expand(c["ny"], c["nx"])
    return _conservative(rho, [r.uniform(0.5, 1.0) * s, v], 2.5 * torch.ones_like(rho), 1.4)


def _tgv(c, r) -> torch.Tensor:
    """Taylor-Green vortex with drawn low-mode velocity perturbations."""
    X, Y, Z = _axis(c["nx"], TWO_PI)[None, None, :], _axis(c["ny"], TWO_PI)[None, :, None], \
        _axis(c["nz"], TWO_PI)[:, None, None]
    ph = [r.uniform(0.0, TWO_PI) for _ in range(6)]
    am = [r.uniform(0.02, 0.1) for _ in range(3)]
    u = torch.sin(X) * torch.cos(Y) * torch.cos(Z) + am[0] * torch.sin(Y + ph[0]) * torch.cos(2 * Z + ph[1])
    v = -torch.cos(X) * torch.sin(Y) * torch.cos(Z) + am[1] * torch.sin(2 * Z + ph[2]) * torch.cos(X + ph[3])
    w = am[2] * torch.sin(X + ph[4]) * torch.cos(2 * Y + ph[5])
    p = 100.0 / 1.4 + (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0) / 16.0
    return _conservative(torch.ones_like(u), [u, v, w], p, 1.4)


def _mhd_state(rho, u, p, B, gamma) -> torch.Tensor:
    u, B = [q.expand_as(rho) for q in u], [q.expand_as(rho) for q in B]
    E = p / (gamma - 1.0) + 0.5 * rho * sum(q * q for q in u) + 0.5 * sum(q * q for q in B)
    return torch.stack([rho] + [rho * q for q in u] + [E] + B)


def _orszag_tang(c, r) -> torch.Tensor:
    """Orszag-Tang vortex; field strength, phases and a weak out-of-plane field drawn."""
    gamma = _gamma(c)
    x, y = _axis(c["nx"], TWO_PI)[None, :], _axis(c["ny"], TWO_PI)[:, None]
    rho = torch.full((c["ny"], c["nx"]), gamma ** 2, dtype=torch.float64, device=_device())
    B0, a, b = r.uniform(0.8, 1.0), r.uniform(0.0, TWO_PI), r.uniform(0.0, TWO_PI)
    u = [-torch.sin(y + a), torch.sin(x + b), 0.1 * torch.sin(x + a) * torch.sin(y + b)]
    B = [-B0 * torch.sin(y), B0 * torch.sin(2 * x + b), 0.1 * torch.cos(x + y + a)]
    return _mhd_state(rho, u, gamma * torch.ones_like(rho), B, gamma)


def _alfven(c, r) -> torch.Tensor:
    """Circularly polarized Alfven wave along x with drawn transverse structure."""
    gamma = _gamma(c)
    X, Y, Z = _axis(c["nx"], 1.0)[None, None, :], _axis(c["ny"], 1.0)[None, :, None], _axis(c["nz"], 1.0)[:, None, None]
    k, a, b = TWO_PI, r.uniform(0.0, TWO_PI), r.uniform(0.0, TWO_PI)
    b1, e = r.uniform(0.05, 0.15), r.uniform(0.02, 0.05)
    rho = 1.0 + e * torch.sin(k * X + a) * torch.cos(k * Y) * torch.cos(k * Z + b)
    by = b1 * torch.cos(k * X) + e * torch.sin(k * (X + Z) + a)
    bz = b1 * torch.sin(k * X) + e * torch.cos(k * (X - Y) + b)
    bx = 1.0 + e * torch.sin(k * (Y + Z) + b)
    return _mhd_state(rho, [e * torch.cos(k * Z + a), -by, -bz], 0.1 + 0.0 * rho, [bx, by, bz], gamma)


def _lgl_axis(n: int, length: float) -> Tuple[np.ndarray, np.ndarray, np.ndarray]:
    """LGL nodes ascending on [0, length], weights of [-1, 1] and the
    differentiation matrix, float64: interior nodes from the Jacobi(1, 1)
    matrix's eigenvalues with one Newton sweep on P'_{n-1}."""
    p = n - 1

    def legendre(x):
        P0, P1 = np.ones_like(x), x.copy()
        for k in range(2, p + 1):
            P0, P1 = P1, ((2 * k - 1) * x * P1 - (k - 1) * P0) / k
        return P0, P1  # P_{p-1}, P_p

    k = np.arange(1, n - 2, dtype=np.float64)
    off = np.sqrt(k * (k + 2) / ((2 * k + 1) * (2 * k + 3)))
    y = np.linalg.eigvalsh(np.diag(off, 1) + np.diag(off, -1))
    for _ in range(2):
        Pm, P = legendre(y)
        dP = p * (Pm - y * P) / (1.0 - y * y)
        y = y - dP * (1.0 - y * y) / (2.0 * y * dP - p * (p + 1) * P)
    y = np.concatenate([[-1.0], 0.5 * (y - y[::-1]), [1.0]])
    P = legendre(y)[1]
    diff = y[:, None] - y[None, :]
    np.fill_diagonal(diff, 1.0)
    D = (P[:, None] / P[None, :]) / diff
    np.fill_diagonal(D, 0.0)
    np.fill_diagonal(D, -D.sum(axis=1))
    return (1.0 + y) * (length / 2.0), 2.0 / (p * n * P * P), D * (2.0 / length)


def _lgl_filter(n: int, length: float) -> np.ndarray:
    x, w, _ = _lgl_axis(n, length)
    V = np.polynomial.legendre.legvander(x * (2.0 / length) - 1.0, n - 1)
    k = np.arange(n, dtype=np.float64)
    sigma = np.exp(-FILTER["alpha"] * (k / (n - 1)) ** FILTER["p"])
    return (V * (sigma * (2.0 * k + 1.0) / 2.0)) @ V.T * w[None, :]


def _pulse(c, r) -> torch.Tensor:
    """Acoustic pulse between walls; centre, width and amplitude drawn."""
    x, y = (torch.as_tensor(_lgl_axis(n, 2.0)[0] - 1.0, device=_device()) for n in (c["nx"], c["ny"]))
    cx, cy = r.uniform(-0.3, 0.3), r.uniform(-0.3, 0.3)
    r2 = (x[None, :] - cx) ** 2 + (y[:, None] - cy) ** 2
    rho = 1.0 + r.uniform(0.005, 0.02) * torch.exp(-r2 / r.uniform(0.02, 0.05))
    u = r.uniform(0.005, 0.02) * torch.sin(math.pi * x)[None, :] * torch.cos(math.pi * y)[:, None]
    return _conservative(rho, [u, torch.zeros_like(rho)], rho ** 1.4 / 1.4, 1.4)


def _inputs(c, seed: int) -> torch.Tensor:
    """Initial states, float32, (ncomp, *shape) or (batch, ncomp, *shape)."""
    make = {("euler", 1): _sod, ("euler", 2): _khi, ("euler", 3): _tgv, ("mhd", 2): _orszag_tang,
            ("mhd", 3): _alfven, ("lgl", 2): _pulse}[(c["kind"], _ndim(c))]
    r = np.random.RandomState(seed % (1 << 31))
    U = [make(c, r).to(torch.float32) for _ in range(c["batch"])]
    return (U[0] if c["batch"] == 1 else torch.stack(U)).contiguous()


def _speed(c, U: torch.Tensor) -> torch.Tensor:
    """CFL wave speed per solve, float64; U (batch, ncomp, ...)."""
    d, g = _ndim(c), _gamma(c)
    rho = U[:, 0]
    if c["kind"] == "mhd":
        u = [U[:, i] / rho for i in (1, 2, 3)]
        b2 = sum(U[:, i] ** 2 for i in (5, 6, 7))
        p = (g - 1.0) * (U[:, 4] - 0.5 * rho * sum(q * q for q in u) - 0.5 * b2)
        um, a = torch.stack([q.abs() for q in u[:d]]).amax(0), torch.sqrt((g * p + b2) / rho)
    else:
        u = [U[:, 1 + i] / rho for i in range(d)]
        p = (g - 1.0) * (U[:, d + 1] - 0.5 * rho * sum(q * q for q in u))
        um = torch.stack([q.abs() for q in (u[:1] if d == 2 else u)]).amax(0)
        a = torch.sqrt(g * p / rho)
    return (um + a).flatten(1).amax(1)


def _hmin(c) -> float:
    if c["kind"] == "lgl":
        return min(float(np.diff(_lgl_axis(n, 2.0)[0]).min()) for n in (c["nx"], c["ny"]))
    return min(L / n for n, L in zip(_shape(c), _lengths(c)))


def _time_plan(c, U: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """Per solve: a fixed step at half the CFL limit, and an end time inside the
    last launched step (the CFL step may shrink as the shock tube starts)."""
    V = U if c["batch"] > 1 else U[None]
    dt = _cfl(c) * _hmin(c) / _speed(c, V.double())
    return 0.5 * dt, dt * (0.4 * c["steps"] if _ndim(c) == 1 else c["steps"] - 0.6)


# ------------------------------------------------------------------ the pass
def _solver(c):
    from phrike_gb300 import equations as E, grid as G, solver as S
    d, fp = _ndim(c), dict(FILTER) if c["filter"] else None
    if c["kind"] == "lgl":
        g = G.Grid2D(c["nx"], c["ny"], 2.0, 2.0, basis_x="legendre", basis_y="legendre", filter_params=fp,
                     gemm_precision=c["precision"])
        return S.SpectralSolver2D(g, E.EulerEquations2D(gamma=1.4), scheme=c["scheme"], cfl=_cfl(c))
    n = [v for v in (c["nx"], c["ny"], c["nz"]) if v]
    g = (G.Grid1D, G.Grid2D, G.Grid3D)[d - 1](*n, *reversed(_lengths(c)), filter_params=fp)
    if c["kind"] == "mhd":
        g.mhd_config = {}
        eq = (E.MHDEquations2D, E.MHDEquations3D)[d - 2](gamma=_gamma(c))
        return (S.SpectralSolverMHD2D, S.SpectralSolverMHD3D)[d - 2](g, eq, scheme=c["scheme"], cfl=_cfl(c))
    eq = (E.EulerEquations1D, E.EulerEquations2D, E.EulerEquations3D)[d - 1](gamma=_gamma(c))
    return (S.SpectralSolver1D, S.SpectralSolver2D, S.SpectralSolver3D)[d - 1](g, eq, scheme=c["scheme"], cfl=_cfl(c))


def prepare(case, seed):
    U = _inputs(case, seed)
    dt, tend = _time_plan(case, U)
    state = {"case": case, "U": U, "dt": float(dt.min()), "t_end": float(tend.min())}
    if case["call"] in ("step", "run"):
        state["solver"] = _solver(case)
    else:
        from phrike_gb300.engine import Plan
        state["plan"] = Plan(_shape(case), _lengths(case), gamma=_gamma(case), cfl=_cfl(case), nsolve=case["batch"],
                             filter_params=dict(FILTER) if case["filter"] else None, scheme=case["scheme"])
        state["t_ends"] = tend.contiguous()
    return state


def run(state):
    case, U = state["case"], state["U"]
    if case["call"] == "step":
        return state["solver"].step(U, state["dt"])
    if case["call"] == "run":
        s = state["solver"]
        s.run(U, 0.0, state["t_end"], output_interval=0.5 * state["t_end"])
        return s.U
    V = U.clone()
    if case["call"] == "fixed":
        return state["plan"].run_(V, case["steps"], state["dt"])
    t = torch.zeros(case["batch"], dtype=torch.float64, device=V.device)
    return state["plan"].run_cfl_(V, case["steps"], t, state["t_ends"])


# ------------------------------------------------------------------ what a pass needs
def work(case):
    d, nc = _ndim(case), _ncomp(case)
    cells = case["batch"] * math.prod(_shape(case))
    stages = case["steps"] * (2 if case["scheme"] == "rk2" else 4)
    if case["kind"] == "lgl":
        flops = stages * nc * cells * 2.0 * (case["nx"] + case["ny"])
    else:
        # distinct flux fields in, one transform back per component, real transforms
        nf = 2 * d + d * (d + 1) // 2 if case["kind"] == "euler" else {2: 13, 3: 18}[d]
        flops = stages * (nf + nc) * cells * 2.5 * math.log2(max(2, math.prod(_shape(case))))
    return {"bytes": 8.0 * nc * cells, "flops": flops}


# ------------------------------------------------------------------ float64 restatement
class _Fourier:
    """Masked, filtered spectral operators of a periodic box by full N-D transforms."""

    def __init__(self, c):
        self.c, self.d, self.shape = c, _ndim(c), _shape(c)
        self.axes = tuple(range(-self.d, 0))
        self.k, self.mult = [], 1.0
        for a, (n, L) in enumerate(zip(self.shape, _lengths(c))):
            j = np.fft.fftfreq(n) * n
            m = (np.abs(j) <= n // 3).astype(float)
            if c["filter"]:
                m = m * np.exp(-FILTER["alpha"] * (np.abs(j) / np.abs(j).max()) ** FILTER["p"])
            view = [1] * self.d
            view[a] = n
            self.k.append(torch.as_tensor(2.0 * np.pi * np.fft.fftfreq(n, d=L / n), device=_device()).reshape(view))
            self.mult = self.mult * torch.as_tensor(m, device=_device()).reshape(view)

    def divergence(self, fluxes):
        """sum over directions (x first) of the masked derivative of each flux."""
        out = []
        for comp in zip(*fluxes):
            s = 0.0
            for a, F in enumerate(comp):
                s = s + 1j * self.k[self.d - 1 - a] * torch.fft.fftn(F, dim=self.axes)
            out.append(torch.fft.ifftn(s * self.mult, dim=self.axes).real)
        return torch.stack(out, dim=1)

    def filt(self, U):
        return torch.stack([torch.fft.ifftn(torch.fft.fftn(U[:, i], dim=self.axes) * self.mult, dim=self.axes).real
                            for i in range(U.shape[1])], dim=1)

    def project(self, B):
        """Leray projection of the in-box field components (x first)."""
        F = [torch.fft.fftn(b, dim=self.axes) for b in B]
        for f in F:
            for a, n in enumerate(self.shape):
                if n % 2 == 0:
                    f.narrow(a - self.d, n // 2, 1).zero_()
        ks = [self.k[self.d - 1 - a] for a in range(self.d)]
        k2 = sum(k * k for k in ks)
        coef = sum(k * f for k, f in zip(ks, F)) / torch.where(k2 == 0.0, torch.ones_like(k2), k2)
        return [torch.fft.ifftn(f - k * coef, dim=self.axes).real for k, f in zip(ks, F)]


def _euler_fluxes(U, d, g):
    rho = U[:, 0]
    u = [U[:, 1 + i] / rho for i in range(d)]
    E = U[:, d + 1]
    p = (g - 1.0) * (E - 0.5 * rho * sum(q * q for q in u))
    return [[U[:, 1 + a]] + [U[:, 1 + a] * u[b] + (p if a == b else 0.0) for b in range(d)] + [(E + p) * u[a]]
            for a in range(d)]


def _mhd_fluxes(U, d, g):
    rho, E = U[:, 0], U[:, 4]
    u, B = [U[:, i] / rho for i in (1, 2, 3)], [U[:, i] for i in (5, 6, 7)]
    b2 = sum(b * b for b in B)
    ps = (g - 1.0) * (E - 0.5 * rho * sum(q * q for q in u) - 0.5 * b2) + 0.5 * b2
    uB = sum(q * b for q, b in zip(u, B))
    return [[U[:, 1 + a]] + [U[:, 1 + a] * u[b] - B[a] * B[b] + (ps if a == b else 0.0) for b in range(3)]
            + [(E + ps) * u[a] - B[a] * uB] + [u[a] * B[b] - u[b] * B[a] for b in range(3)] for a in range(d)]


def _floors(U, d, g, floors, mhd):
    """primitive -> floors -> conservative (identity where no floor acts)."""
    rho, m = U[:, 0], 3 if mhd else d
    kin = 0.5 * sum((U[:, 1 + i] / rho) ** 2 for i in range(m))
    mag = 0.5 * sum(U[:, i] ** 2 for i in (5, 6, 7)) if mhd else 0.0
    p = (g - 1.0) * (U[:, m + 1] - rho * kin - mag)
    rc, pc = rho.clamp(min=floors[0]), p.clamp(min=floors[1])
    V = U.clone()
    V[:, 0], V[:, m + 1] = rc, pc / (g - 1.0) + rc * kin + mag
    for i in range(m):
        V[:, 1 + i] = U[:, 1 + i] / rho * rc
    return V


def _walls(U):
    for dst, src in ((0, 1), (-1, -2)):
        U[:, :, :, dst] = U[:, :, :, src]
        U[:, 1, :, dst] = 0.0
    for dst, src in ((-1, -2), (0, 1)):
        U[:, :, dst, :] = U[:, :, src, :]
        U[:, 2, dst, :] = 0.0
    return U


class _Exact:
    """One step of the schemes, U (batch, ncomp, *shape) float64, dt (batch,)."""

    def __init__(self, c):
        self.c, self.d, self.g = c, _ndim(c), _gamma(c)
        self.lgl, self.mhd = c["kind"] == "lgl", c["kind"] == "mhd"
        if self.lgl:
            self.D = [torch.as_tensor(_lgl_axis(n, 2.0)[2], device=_device()) for n in (c["nx"], c["ny"])]
            self.F = [torch.as_tensor(_lgl_filter(n, 2.0), device=_device()) for n in (c["nx"], c["ny"])]
        else:
            self.box = _Fourier(c)
        self.floors = (1e-10, 1e-12) if (self.mhd or self.d == 1) else (1e-8, 1e-10)

    def rhs(self, U):
        if self.lgl:
            _walls(U)
            Fx, Fy = (torch.stack(f, dim=1) for f in _euler_fluxes(U, 2, self.g))
            return -(Fx @ self.D[0].T + self.D[1] @ Fy)
        return -self.box.divergence((_mhd_fluxes if self.mhd else _euler_fluxes)(U, self.d, self.g))

    def after(self, U):
        """After every stage: floors (none in 3D Euler), MHD projection."""
        if self.mhd or self.d < 3:
            U = _floors(U, self.d, self.g, self.floors, self.mhd)
        return self.project(U) if self.mhd else U

    def project(self, U):
        """B projected, the thermal pressure held fixed."""
        V = U.clone()
        for i, b in enumerate(self.box.project([U[:, 5 + i] for i in range(self.d)])):
            V[:, 5 + i] = b
        V[:, 4] += 0.5 * sum(V[:, i] ** 2 - U[:, i] ** 2 for i in (5, 6, 7))
        return V

    def step(self, U, dt):
        h = dt.reshape((-1,) + (1,) * (U.dim() - 1))
        if self.c["scheme"] == "rk2":
            V = self.after(U + 0.5 * h * self.rhs(U))
            V = self.after(U + h * self.rhs(V))
        else:
            k = self.rhs(U)
            s = k
            for w, a in ((2.0, 0.5), (2.0, 0.5), (1.0, 1.0)):
                k = self.rhs(self.after(U + a * h * k))
                s = s + w * k
            V = self.after(U + (h / 6.0) * s)
        if self.lgl:
            if self.c["filter"]:
                V = self.F[1] @ (V @ self.F[0].T)
            return _walls(V)
        V = self.box.filt(V)
        if self.d == 1:
            V = self.box.filt(V)
        return self.project(V) if self.mhd else V


def exact(case, seed):
    U0 = _inputs(case, seed)
    fixed, tend = _time_plan(case, U0)
    U = (U0 if case["batch"] > 1 else U0[None]).double()
    if case["kind"] == "lgl":
        U = U.clone()
    solve = _Exact(case)
    if case["call"] in ("step", "fixed"):
        for _ in range(case["steps"] if case["call"] == "fixed" else 1):
            U = solve.step(U, fixed.min().expand(U.shape[0]))
    else:
        # run: one solve to t_end, however many steps it takes; cfl: at most `steps`
        t = torch.zeros_like(tend)
        n = 0
        while bool((t < tend - 1e-12).any()) and (case["call"] == "run" or n < case["steps"]):
            dt = torch.minimum(_cfl(case) * _hmin(case) / _speed(case, U), tend - t)
            live = t < tend - 1e-12
            V = solve.step(U, torch.where(live, dt, torch.zeros_like(dt)))
            U = torch.where(live.reshape((-1,) + (1,) * (U.dim() - 1)), V, U)
            t = torch.where(live, t + dt, t)
            n += 1
    return U if case["batch"] > 1 else U[0]
