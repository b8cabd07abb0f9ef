"""Whole-step 1D kernel (csrc/line1d.cuh) against the float64 oracle at every
power of two from 8 (the kernel below it) to 4096: the fused pass is radix 4
or 8 by parity, from 64 threads the time step is computed by a warp of its
own, from 2048 points the state lives in shared memory.

Bound: five transforms' rounding per step, each at most about 4 eps per pass
over 12 passes in norm, 5 * 48 * 6e-8 = 1.4e-5 per step at worst and far less
on average (rounding errors of different passes do not align); the
repository's bar of 1e-5 for states is asked for over 6 steps.  Gravity,
cadence and midpoint steps share the code path."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [8, 16, 32, 64, 128, 256, 512, 1024, 2048, 4096]


def state(n, seed):
    r = np.random.RandomState(seed)
    x = np.arange(n) / n * 2 * np.pi
    f = lambda m, a: m + a * sum(np.cos(k * x + r.uniform(0, 6)) / k for k in (1, 2, 3) if k < n // 2) \
        + 0.02 * a * r.standard_normal(n)
    rho, u, p = f(1.0, 0.2), f(0.1, 0.3), f(2.0, 0.3)
    return np.stack([rho, rho * u, p / 0.4 + 0.5 * rho * u * u])


def check(got, ref):
    for c in range(3):
        assert np.linalg.norm(got[c] - ref[c]) / np.linalg.norm(ref[c]) < 1e-5, c


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("scheme,interval,gx", [("rk4", 1, 0.0), ("rk4", 2, 1.5), ("rk2", 1, 0.0)])
def test_fixed_steps(n, scheme, interval, gx):
    from oracle import spectral as O
    from phrike_gb300.engine import Plan
    fp = {"enabled": True, "p": 8, "alpha": 36.0, "interval": interval}
    U0 = state(n, 1).astype(np.float32)
    s = O.EulerSolver(O.FourierBox((n,), (1.0,), filter_enabled=True), filter_interval=interval, scheme=scheme,
                      gravity=(gx,) if gx else None)
    dt = 0.2 * s.compute_dt(U0.astype(np.float64))
    plan = Plan((n,), (1.0,), filter_params=fp, scheme=scheme, gravity=(gx,))
    U = torch.as_tensor(U0, device="cuda")
    plan.run_(U, 5, dt)
    plan.step_(U, dt)
    ref = U0.astype(np.float64)
    for _ in range(6):
        ref = s.step(ref, dt)
    check(U.double().cpu().numpy(), ref)


@pytest.mark.parametrize("n", SIZES)
def test_cfl_batch(n):
    """Solves that never start, end early or run through the chunk; each has
    the bits of the same solve alone."""
    from oracle import spectral as O
    from phrike_gb300.engine import Plan
    fp = {"enabled": True, "p": 8, "alpha": 36.0}
    U0 = np.stack([state(n, i) for i in range(3)]).astype(np.float32)
    s = O.EulerSolver(O.FourierBox((n,), (1.0,), filter_enabled=True), cfl=0.4)
    tend = [0.0, 1.5 * s.compute_dt(U0[1].astype(np.float64)), 10.0]
    f64 = dict(dtype=torch.float64, device="cuda")
    plan = Plan((n,), (1.0,), filter_params=fp, cfl=0.4, nsolve=3)
    U, t = torch.as_tensor(U0, device="cuda"), torch.zeros(3, **f64)
    plan.run_cfl_(U, 4, t, torch.as_tensor(tend, **f64))
    assert plan.steps_done() == [0, 2, 4]
    one = Plan((n,), (1.0,), filter_params=fp, cfl=0.4)
    for i in range(3):
        V, ti = torch.as_tensor(U0[i], device="cuda"), torch.zeros(1, **f64)
        one.run_cfl_(V, 4, ti, torch.as_tensor(tend[i:i + 1], **f64))
        assert torch.equal(V, U[i]) and float(ti) == float(t[i])
        ref, tr, _ = s.run(U0[i].astype(np.float64), 0.0, tend[i], max_steps=4)
        check(U[i].double().cpu().numpy(), ref)
        assert abs(float(t[i]) - tr) <= 1e-6 * tr
