"""N tiles of the tcgen05 LGL contractions (ps_plan_desc.umma_n_tile): the four
values select four kernels in the steps by even and odd parts (csrc/lgl_eo.cu)
and four in the full-size contractions of the right-hand side, gravity and
filter cadences above 1 (csrc/lgl_tc.cu).  Every output is the same dot product
in each, so states are compared by bits; one tile of each kind is held to the
oracle by the other LGL tests, and each tile once here.

Bound against the oracle: as tests/test_gpu_lgl_even_odd.py, 1e-5."""
import numpy as np
import pytest

from test_gpu_batch_bits import same_alone
from test_gpu_lgl_even_odd import check, state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TILES = (64, 128, 176, 256)
FP = {"enabled": True, "p": 8, "alpha": 36.0}


def states(nx, ny, nsolve):
    from oracle import lgl as L
    ax, ay = L.LGLAxis(nx, 2.0), L.LGLAxis(ny, 2.0)
    return np.stack([state(ax, ay, i) for i in range(nsolve)])


def outputs(nx, ny, nsolve, run, **kw):
    from phrike_gb300.engine import Plan
    U0 = torch.as_tensor(states(nx, ny, nsolve).astype(np.float32), device="cuda")
    outs = []
    for nt in TILES:
        plan = Plan((ny, nx), (2.0, 2.0), basis="legendre", gemm_precision="bf16x3", nsolve=nsolve, umma_n_tile=nt, **kw)
        outs.append(run(plan, U0.clone()))
        assert plan.status() == 0
    return outs


# node pairs on both sides of a tile's end: 48, 64, 80, 144 and the last
# 64-wide block of a dot product
@pytest.mark.parametrize("nx,ny,nsolve", [(3, 3, 1), (17, 16, 3), (96, 97, 1), (128, 129, 2), (161, 160, 1),
                                          (288, 289, 1), (300, 300, 1), (33, 290, 2)])
@pytest.mark.parametrize("filt", [False, True])
def test_step_tiles(nx, ny, nsolve, filt):
    from oracle import lgl as L
    fp = dict(FP, enabled=filt)
    s = L.LGLSolver2D(nx, ny, filter_params=fp, cfl=0.3)
    ref = states(nx, ny, nsolve)[0].astype(np.float32).astype(np.float64)
    dt = 0.5 * s.compute_dt(ref)
    outs = outputs(nx, ny, nsolve, lambda p, U: p.run_(U, 3, dt), filter_params=fp)
    for V in outs[1:]:
        assert torch.equal(outs[0], V)
    for _ in range(3):
        ref = s.step(ref, dt)
    check(outs[0][0].double().cpu().numpy(), ref)


@pytest.mark.parametrize("kw", [dict(gravity=(0.2, -0.4)), dict(filter_params=dict(FP, interval=2)), "rhs"], ids=str)
@pytest.mark.parametrize("nx,ny,nsolve", [(65, 65, 2), (129, 64, 1), (63, 177, 1), (257, 40, 1)])
def test_full_size_tiles(nx, ny, nsolve, kw):
    if kw == "rhs":
        outs = outputs(nx, ny, nsolve, lambda p, U: p.rhs(U))
    else:
        outs = outputs(nx, ny, nsolve, lambda p, U: p.run_(U, 3, 1e-5), **kw)
    for V in outs[1:]:
        assert torch.equal(outs[0], V)


# the plan's own choice: 48 for each solve alone; 64, 80 and 144 for the batch
@pytest.mark.parametrize("n,nsolve", [(97, 8), (129, 8), (257, 16)])
@pytest.mark.parametrize("prec", ["fp32", "bf16x3"])
@pytest.mark.parametrize("filt", [False, True])
def test_batches_choose_other_tiles_than_solves_alone(n, nsolve, prec, filt):
    same_alone(states(n, n, 3), nsolve, lambda p, U: p.run_(U, 2, 1e-5), basis="legendre", gemm_precision=prec,
               filter_params=dict(FP, enabled=filt))
