"""Stepping on the truncated-spectra passes (csrc/spectral.cuh) against the
float64 oracle over the shapes where their index arithmetic can go wrong: the
shortest and longest axes in either place, unequal axes, batches whose solves
end at different times (one before the first step), both schemes, and filter
cadences that skip steps.

Bound: each RK stage rounds the state to float32 and carries the transforms'
rounding, at most about 8 eps per stage; over at most 4 steps of 4 stages that
is 16 * 8 * 6e-8 = 8e-6 of a field's norm, so 1e-5 (the repository's bar for
states) holds.  Momentum and magnetic field are measured as vectors."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FP = {"enabled": True, "p": 8, "alpha": 36.0}


def euler_state(shape, seed):
    """Smooth flow with content beyond the 2/3 mask."""
    r = np.random.RandomState(seed)
    d = len(shape)
    x = np.meshgrid(*[np.arange(n) * 2 * np.pi / n for n in shape], indexing="ij")

    def field(mean, amp):
        f = np.full(shape, mean)
        for _ in range(4):
            k = [r.randint(0, min(4, n // 2)) for n in shape]
            f = f + amp * np.cos(sum(a * b for a, b in zip(k, x)) + r.uniform(0, 6.28)) / 4
        return f + 0.02 * amp * r.standard_normal(shape)

    rho, u, p = field(1.0, 0.2), [field(0.0, 0.3) for _ in range(d)], field(2.0, 0.3)
    return np.stack([rho] + [rho * v for v in u] + [p / 0.4 + 0.5 * rho * sum(v * v for v in u)])


def mhd_state(shape, seed):
    U = euler_state(shape, seed)
    r = np.random.RandomState(seed + 1)
    d = len(shape)
    m = [U[1 + i] for i in range(d)] + [0.1 * U[0]] * (3 - d)
    B = [0.4 + 0.2 * np.roll(U[1 + i % d], i + 1, axis=0) + 0.01 * r.standard_normal(shape) for i in range(3)]
    E = 2.0 / (2.0 / 3.0) + 0.5 * sum(v * v for v in m) / U[0] + 0.5 * sum(b * b for b in B)
    return np.stack([U[0]] + m + [E] + B)


def check(got, ref, d, mhd):
    groups = [[0], list(range(1, 4)), [4], [5, 6, 7]] if mhd else [[0], list(range(1, d + 1)), [d + 1]]
    for g in groups:
        err = np.linalg.norm(got[g] - ref[g]) / np.linalg.norm(ref[g])
        assert err < 1e-5, (g, err)


SHAPES2 = [(8, 8), (8, 16), (16, 8), (32, 64), (512, 8), (8, 512), (1024, 16), (16, 1024), (128, 256)]
# axes of 2^a 3^b 5^c points (csrc/mr_spec.cu): odd, prime powers, the longest,
# in either place and beside a power of two
SHAPES2 += [(45, 64), (64, 45), (3, 40), (40, 6), (250, 96), (96, 250), (3645, 8), (8, 3645), (2048, 12), (12, 2048),
            (4096, 10), (10, 4096), (27, 25), (360, 480), (16, 3125)]
SHAPES3 = [(15, 16, 27), (16, 15, 8), (8, 27, 20), (30, 8, 16), (12, 10, 9), (6, 5, 4), (81, 8, 10), (8, 125, 9),
           (10, 9, 1500)]
SHAPES3 += [(8, 8, 8), (8, 16, 32), (32, 8, 16), (16, 64, 8), (64, 8, 8), (8, 8, 512), (8, 512, 8), (256, 8, 8)]


@pytest.mark.parametrize("shape", SHAPES2 + SHAPES3, ids=str)
@pytest.mark.parametrize("scheme,filt,interval", [("rk4", FP, 1), ("rk4", None, 1), ("rk2", FP, 2)])
def test_euler_steps(shape, scheme, filt, interval):
    from oracle import spectral as O
    from phrike_gb300.engine import Plan
    d = len(shape)
    U0 = euler_state(shape, 3).astype(np.float32)
    lengths = tuple(1.0 + 0.5 * i for i in range(d))
    fp = dict(filt, interval=interval) if filt else {"interval": interval}
    box = O.FourierBox(shape, lengths, filter_enabled=bool(filt))
    s = O.EulerSolver(box, filter_interval=interval, scheme=scheme)
    dt = 0.2 * s.compute_dt(U0.astype(np.float64))
    plan = Plan(shape, lengths, filter_params=fp, scheme=scheme)
    U = torch.as_tensor(U0, device="cuda")
    plan.run_(U, 3, dt)
    ref = U0.astype(np.float64)
    for _ in range(3):
        ref = s.step(ref, dt)
    check(U.double().cpu().numpy(), ref, d, False)
    plan.step_(U, dt)
    check(U.double().cpu().numpy(), s.step(ref, dt), d, False)
    assert plan.status() == 0


@pytest.mark.parametrize("shape", [(8, 8), (16, 8), (8, 64), (64, 32), (512, 16), (16, 512), (8, 8, 8), (16, 8, 32),
                                   (8, 32, 16), (8, 8, 256), (256, 8, 8)], ids=str)
@pytest.mark.parametrize("options", [{}, {"project_each_substage": False}, {"divergence_clean": "none"}], ids=str)
@pytest.mark.parametrize("interval", [1, 2])
def test_mhd_steps(shape, options, interval):
    from oracle import mhd as M
    from phrike_gb300.engine import Plan
    d = len(shape)
    U0 = mhd_state(shape, 5).astype(np.float32)
    fp = dict(FP, interval=interval)
    kw = dict(gamma=5.0 / 3.0, filter_params=fp, **options)
    s = M.MHDSolver2D(*reversed(shape), 1.0, 1.0, **kw) if d == 2 else M.MHDSolver3D(*reversed(shape), 1.0, 1.0, 1.0, **kw)
    dt = 0.2 * 0.3 / max(shape) / M.max_wave_speed_3d(U0.astype(np.float64), 5.0 / 3.0)
    plan = Plan(shape, (1.0,) * d, gamma=5.0 / 3.0, filter_params=fp, equations="mhd", mhd_config=options)
    U = torch.as_tensor(U0, device="cuda")
    plan.run_(U, 3, dt)
    ref = U0.astype(np.float64)
    for _ in range(3):
        ref = s.step(ref, dt)
    check(U.double().cpu().numpy(), ref, d, True)


@pytest.mark.parametrize("shape", [(16, 8), (64, 64), (256, 32), (8, 16, 8), (45, 60), (64, 90), (9, 16, 10)], ids=str)
def test_euler_cfl_batch(shape):
    """Three solves of one plan: one already at its end, one that ends inside
    the chunk, one that runs through it."""
    from oracle import spectral as O
    from phrike_gb300.engine import Plan
    d = len(shape)
    U0 = np.stack([euler_state(shape, i) for i in range(3)]).astype(np.float32)
    lengths = (1.0,) * d
    s = O.EulerSolver(O.FourierBox(shape, lengths, filter_enabled=True), cfl=0.3)
    dts = [s.compute_dt(U0[i].astype(np.float64)) for i in range(3)]
    tend = [0.0, 1.5 * dts[1], 100.0]
    plan = Plan(shape, lengths, filter_params=FP, cfl=0.3, nsolve=3)
    U = torch.as_tensor(U0, device="cuda")
    t = torch.zeros(3, dtype=torch.float64, device="cuda")
    plan.run_cfl_(U, 4, t, torch.as_tensor(tend, dtype=torch.float64, device="cuda"))
    got = U.double().cpu().numpy()
    np.testing.assert_allclose(got[0], U0[0], rtol=1e-6, atol=1e-6)
    for i in (1, 2):
        ref, tr, _ = s.run(U0[i].astype(np.float64), 0.0, tend[i], max_steps=4)
        check(got[i], ref, d, False)
        assert abs(float(t[i]) - tr) < 1e-6 * tr
    assert plan.steps_done() == [0, 2, 4]
