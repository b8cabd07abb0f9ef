"""The x rows of the truncated-spectra steps run in one warp per row group
(k_spec_x, csrc/spectral.cuh) or in several warps that share them (k_spec_xs:
MHD, and Euler where the rows are few).  A large Euler batch takes the first
kernel and each of its solves alone the second; the CTAs of a large MHD batch
walk over several tiles of rows, those of one solve take one tile each.  All
run the same operations per value, so their states differ by rounding only.

Bound: both are within 8e-6 of exact arithmetic over these steps (16 stages of
8 eps), and they share all but the contraction of products and sums, so half of
the sum of the two is allowed: 8e-6 of a field's norm."""
import numpy as np
import pytest

from test_gpu_truncated_spectra import euler_state, mhd_state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# rows times threads per row beyond 8 warps on each of 152 SMs
BATCHES = [((9, 8), 2500), ((8, 16), 1300), ((8, 32), 1300), ((64, 64), 80), ((8, 128), 640), ((8, 256), 320),
           ((8, 512), 160), ((8, 8, 8), 320), ((8, 9, 128), 72)]


@pytest.mark.parametrize("equations", ["euler", "mhd"])
@pytest.mark.parametrize("shape,nsolve", BATCHES, ids=str)
def test_batch_equals_single_solves(shape, nsolve, equations):
    from phrike_gb300.engine import Plan
    mhd = equations == "mhd"
    if mhd and 9 in shape:
        shape = tuple(8 if n == 9 else n for n in shape)
    d = len(shape)
    make = mhd_state if mhd else euler_state
    base = [make(shape, i) for i in range(3)]
    U0 = np.stack([base[i % 3] for i in range(nsolve)]).astype(np.float32)
    kw = dict(filter_params={"enabled": True, "p": 8, "alpha": 36.0}, equations=equations)
    if mhd:
        kw["mhd_config"] = {}
    dt = 0.02 / max(shape)
    batch = Plan(shape, (1.0,) * d, nsolve=nsolve, **kw)
    U = torch.as_tensor(U0, device="cuda")
    batch.run_(U, 3, dt)
    got = U.double().cpu().numpy()
    single = Plan(shape, (1.0,) * d, **kw)
    for i in (0, 1, nsolve - 1):
        V = torch.as_tensor(U0[i], device="cuda")
        single.run_(V, 3, dt)
        ref = V.double().cpu().numpy()
        groups = [[0], [1, 2, 3], [4], [5, 6, 7]] if mhd else [[0], list(range(1, d + 1)), [d + 1]]
        for g in groups:
            err = np.linalg.norm(got[i][g] - ref[g]) / np.linalg.norm(ref[g])
            assert err < 8e-6, (i, g, err)
    assert batch.status() == 0
