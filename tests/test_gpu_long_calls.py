"""Many steps in one call of the truncated-spectra passes (csrc/ps_api.cu,
steps_spec), which leave out work that is an identity in exact arithmetic: what
float32 rounding leaves behind must not grow with the length of the call."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def outside_mask(U):
    """Norm of each field's spectrum outside the 2/3 mask, relative to the field's."""
    F = torch.fft.fftn(U.double(), dim=(1, 2, 3))
    n = U.shape[-1]
    k = torch.fft.fftfreq(n, 1.0 / n, device=U.device).abs() <= n // 3
    keep = k[:, None, None] & k[None, :, None] & k[None, None, :]
    power = F.abs().pow(2)
    return ((power * ~keep).sum((1, 2, 3)) / power.sum((1, 2, 3))).sqrt()


@pytest.mark.parametrize("steps", [7, 8, 9, 200])
def test_mask_filter_over_a_long_call(steps):
    """3D Euler with the mask alone, one call against calls of one step (each
    of which ends with the filter).  The filter acts on every eighth step of a
    call, so a state carries at most 7 roundings beside the filter's own, all
    of about one size: sqrt(8) < 3 of a filtered state's, 4 with a margin.
    States: each is within 3.4e-6 of the oracle after 200 such steps, so 1e-5
    between them."""
    from phrike_gb300 import problems
    from phrike_gb300.engine import Plan
    n = 32
    U0 = torch.as_tensor(problems.taylor_green_3d(n), dtype=torch.float32, device="cuda").contiguous()
    one, each = U0.clone(), U0.clone()
    plan = Plan((n,) * 3, (2 * np.pi,) * 3)
    plan.run_(one, steps, 0.3 / n)
    for _ in range(steps):
        plan.step_(each, 0.3 / n)
    ratio = (outside_mask(one) / outside_mask(each)).cpu().numpy()
    assert (ratio < 4.0).all(), ratio
    for g in ([0], [1, 2, 3], [4]):
        assert float((one[g] - each[g]).norm() / each[g].norm()) < 1e-5, g


def orszag_tang(n, d):
    """Orszag-Tang in the x-y plane (gamma 5/3); in 3D with a field along z and velocities that depend on z."""
    x = np.arange(n) * 2 * np.pi / n
    Z, Y, X = np.meshgrid(x if d == 3 else x[:1], x, x, indexing="ij")
    one = np.ones_like(X)
    rho, p = 25 / 9 * one, 5 / 3 * one
    u, v, w = -np.sin(Y) * one, np.sin(X) + 0.3 * np.sin(Z), 0.3 * np.sin(Y) * one * (d == 3)
    bx, by, bz = -np.sin(Y) + 0.2 * np.sin(Z), np.sin(2 * X) * one, 0.5 * one * (d == 3)
    E = p / (2 / 3) + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * (bx * bx + by * by + bz * bz)
    U = np.stack([rho, rho * u, rho * v, rho * w, E, bx, by, bz])
    return U if d == 3 else U[:, 0]


def divergence(U):
    """Root mean square of div B over a 2 pi box, spectral derivatives in float64."""
    d = U.dim() - 1
    total = 0
    for a in range(d):
        axis, n = d - 1 - a, U.shape[d - a]
        k = torch.fft.fftfreq(n, 1.0 / n, device=U.device, dtype=torch.float64)
        k[n // 2] = 0.0
        k = k.reshape([-1 if i == axis else 1 for i in range(d)])
        total = total + torch.fft.ifft(1j * k * torch.fft.fft(U[5 + a].double(), dim=axis), dim=axis).real
    return float(total.pow(2).mean().sqrt())


@pytest.mark.parametrize("n,d", [(128, 2), (32, 3)])
@pytest.mark.parametrize("interval", [1, 50, 1000])
@pytest.mark.parametrize("cfl", [False, True])
def test_divergence_over_a_long_call(n, d, interval, cfl):
    """MHD with projected substages, one call of 200 steps against calls of one
    step, each of which projects the B that its stages start from.  In the long
    call no more than four steps pass without a projection, so the rounding
    divergence of four steps meets that of one: sqrt(4) = 2, 2.5 with a margin.
    (Projecting at the filter's cadence alone leaves up to 23 times as much.)"""
    from phrike_gb300.engine import Plan
    U0 = torch.as_tensor(orszag_tang(n, d), dtype=torch.float32, device="cuda").contiguous()
    kw = dict(gamma=5.0 / 3.0, equations="mhd", mhd_config={}, cfl=0.2,
              filter_params={"enabled": True, "p": 8, "alpha": 36.0, "interval": interval})
    f64 = dict(dtype=torch.float64, device="cuda")
    t, end = torch.zeros(1, **f64), torch.full((1,), 100.0, **f64)

    def advance(plan, U, steps):
        plan.run_cfl_(U, steps, t, end) if cfl else plan.run_(U, steps, 0.15 / n)

    one, each = U0.clone(), U0.clone()
    advance(Plan(U0.shape[1:], (2 * np.pi,) * d, **kw), one, 200)
    t.zero_()
    plan = Plan(U0.shape[1:], (2 * np.pi,) * d, **kw)
    for _ in range(200):
        advance(plan, each, 1)
    assert divergence(one) < 2.5 * divergence(each)
