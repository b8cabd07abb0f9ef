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
