"""LGL x LGL steps by even and odd parts (csrc/lgl_eo.cu) against the float64
oracle: odd and even node counts (a centre line that is its own mirror or
none), the smallest grids (every point beside two walls), unequal axes, one
and several tiles of rows and columns, with and without the filter, both
schemes, and solves of a batch that end at different times.

Bound: the state is stored in float32 (6e-8 of its size per rounding, three
roundings per stage, 16 stages: 3e-6 of a field's norm at worst), the products
keep float32's 24 bits and enter scaled by dt D <= the CFL number < 1.  So 1e-5
holds for density, energy and the momentum vector."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [(3, 3), (4, 3), (3, 5), (5, 4), (16, 17), (33, 64), (65, 40), (96, 97), (129, 130), (258, 33), (31, 260)]


def state(ax, ay, seed):
    r = np.random.RandomState(seed)
    X, Y = np.meshgrid(ax.x - 1.0, ay.x - 1.0, indexing="xy")
    f = lambda m, a: m + a * sum(np.cos(k * X + r.uniform(0, 6)) * np.cos(l * Y + r.uniform(0, 6)) for k, l in
                                 ((1, 0), (0, 1), (1, 2)))
    rho, u, v, p = f(1.0, 0.05), f(0.0, 0.1), f(0.05, 0.1), f(1.0, 0.05)
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])


def check(got, ref):
    for g in ([0], [1, 2], [3]):
        assert np.linalg.norm(got[g] - ref[g]) / np.linalg.norm(ref[g]) < 1e-5, g


@pytest.mark.parametrize("nx,ny", SHAPES)
@pytest.mark.parametrize("prec", ["fp32", "bf16x3"])
@pytest.mark.parametrize("filt,scheme", [(False, "rk4"), (True, "rk4"), (True, "rk2")])
def test_fixed_steps(nx, ny, prec, filt, scheme):
    from oracle import lgl as L
    from phrike_gb300.engine import Plan
    fp = {"enabled": filt, "p": 8, "alpha": 36.0}
    s = L.LGLSolver2D(nx, ny, filter_params=fp, scheme=scheme, cfl=0.3)
    U0 = state(s.ax, s.ay, nx + ny).astype(np.float32)
    dt = 0.5 * s.compute_dt(U0.astype(np.float64))
    plan = Plan((ny, nx), (2.0, 2.0), basis="legendre", gemm_precision=prec, filter_params=fp, scheme=scheme)
    U = torch.as_tensor(U0, device="cuda")
    plan.run_(U, 3, dt)
    plan.step_(U, dt)
    ref = U0.astype(np.float64)
    for _ in range(4):
        ref = s.step(ref, dt)
    check(U.double().cpu().numpy(), ref)
    assert plan.status() == 0


@pytest.mark.parametrize("nx,ny", [(17, 16), (40, 65)])
@pytest.mark.parametrize("filt", [False, True])
def test_cfl_batch(nx, ny, filt):
    from oracle import lgl as L
    from phrike_gb300.engine import Plan
    fp = {"enabled": filt, "p": 8, "alpha": 36.0}
    solvers = [L.LGLSolver2D(nx, ny, filter_params=fp, cfl=0.3) for _ in range(3)]
    U0 = np.stack([state(s.ax, s.ay, i) for i, s in enumerate(solvers)]).astype(np.float32)
    dts = [s.compute_dt(U0[i].astype(np.float64)) for i, s in enumerate(solvers)]
    tend = [0.0, 1.5 * dts[1], 1.0]
    plan = Plan((ny, nx), (2.0, 2.0), basis="legendre", filter_params=fp, cfl=0.3, nsolve=3)
    f64 = dict(dtype=torch.float64, device="cuda")
    U, t = torch.as_tensor(U0, device="cuda"), torch.zeros(3, **f64)
    plan.run_cfl_(U, 3, t, torch.as_tensor(tend, **f64))
    got = U.double().cpu().numpy()
    np.testing.assert_allclose(got[0], U0[0], rtol=1e-6, atol=1e-6)
    for i, steps in ((1, 2), (2, 3)):
        ref, tt = U0[i].astype(np.float64), 0.0
        for _ in range(steps):
            h = min(solvers[i].compute_dt(ref), tend[i] - tt)
            ref, tt = solvers[i].step(ref, h), tt + h
        check(got[i], ref)
        assert abs(float(t[i]) - tt) <= 1e-6 * tt
