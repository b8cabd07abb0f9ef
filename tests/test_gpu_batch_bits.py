"""A solve ends on the same bits alone and in a batch, whatever kernel shapes
the batch's size selects: the Euler x rows in one warp per row group or in
several that share them (csrc/spec_launch.cuh), the MHD projection's tile
widths (csrc/mhd_passes.cuh), the tiles and registers of the filter on
2^a 3^b 5^c axes (csrc/mr_spec.cu), each at sizes on both sides of the choice.
The arithmetic of a value is the same in every shape, so the
tolerance is zero."""
import numpy as np
import pytest

from test_gpu_truncated_spectra import euler_state, mhd_state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FP = {"enabled": True, "p": 8, "alpha": 36.0}


def same_alone(U0, nsolve, run, **kw):
    """run(plan, states) on a batch that repeats the states of U0, and on each alone."""
    from phrike_gb300.engine import Plan
    shape = U0.shape[2:]
    lengths = (1.0,) * len(shape)
    index = torch.arange(nsolve, device="cuda") % len(U0)
    first = torch.as_tensor(U0.astype(np.float32), device="cuda")
    batch = Plan(shape, lengths, nsolve=nsolve, **kw)
    got = run(batch, first[index].contiguous())
    for i in sorted({0, 1, min(2, nsolve - 1), nsolve // 2, nsolve - 1}):
        V = run(Plan(shape, lengths, **kw), first[index[i]].clone())  # (a plan of its own: cadences count its steps)
        assert torch.equal(got[i], V), (i, float((got[i] - V).abs().max()))
    assert batch.status() == 0


@pytest.mark.parametrize("filt,interval", [(None, 1), (FP, 1), (FP, 2)])
@pytest.mark.parametrize("shape,nsolve", [((8, 8), 2500), ((8, 16), 1300), ((8, 32), 1300), ((64, 64), 80),
                                          ((8, 128), 640), ((8, 256), 320), ((512, 512), 3), ((8, 8, 8), 320),
                                          ((64, 64, 64), 2), ((8, 9, 128), 72)], ids=str)
def test_euler_steps(shape, nsolve, filt, interval):
    U0 = np.stack([euler_state(shape, i) for i in range(3)])
    U0[2, -1] *= 0.45  # pressures below zero: the 2D clamp acts
    U0[2, -1] += 0.3
    dt = 0.02 / max(shape)
    same_alone(U0, nsolve, lambda p, U: p.run_(U, 3, dt), filter_params=dict(filt or {}, interval=interval))


@pytest.mark.parametrize("shape,nsolve", [((8, 8), 2500), ((9, 8), 2500), ((8, 16), 1300), ((8, 32), 1300),
                                          ((64, 64), 80), ((8, 128), 640), ((8, 256), 320), ((512, 512), 3),
                                          ((8, 8, 8), 320), ((64, 64, 64), 2)], ids=str)
def test_euler_cfl_steps(shape, nsolve):
    U0 = np.stack([euler_state(shape, i) for i in range(3)])

    def run(plan, U):
        f64 = dict(dtype=torch.float64, device="cuda")
        plan.run_cfl_(U, 3, torch.zeros(plan.nsolve, **f64), torch.full((plan.nsolve,), 1.0, **f64))
        return U

    same_alone(U0, nsolve, run, filter_params=FP, cfl=0.3)


@pytest.mark.parametrize("shape,nsolve", [((8, 8), 2500), ((16, 256), 300), ((256, 16), 300), ((256, 32), 512),
                                          ((64, 64), 80), ((512, 8), 200), ((8, 512), 200), ((1024, 8), 40),
                                          ((16, 16, 16), 40), ((64, 8, 32), 20)], ids=str)
@pytest.mark.parametrize("options", [{}, {"project_each_substage": False}, {"resistivity": 1e-3}], ids=str)
def test_mhd_steps(shape, nsolve, options):
    U0 = np.stack([mhd_state(shape, i) for i in range(3)])
    dt = 0.02 / max(shape)
    same_alone(U0, nsolve, lambda p, U: p.run_(U, 2, dt), filter_params=FP, equations="mhd", mhd_config=options,
               gamma=5.0 / 3.0)


@pytest.mark.parametrize("shape,nsolve", [((9, 8), 2500), ((3, 1000), 200), ((2, 300), 300), ((6, 45), 500),
                                          ((12, 10), 2000), ((96, 90), 64), ((250, 250), 8), ((3, 4096), 40),
                                          ((15, 10, 12), 300), ((30, 30, 30), 8), ((4, 3, 250), 100)], ids=str)
def test_filter_on_mixed_radix_axes(shape, nsolve):
    U0 = np.stack([euler_state(shape, i) for i in range(3)])
    same_alone(U0, nsolve, lambda p, U: p.filter(U), filter_params=FP)


@pytest.mark.parametrize("shape,nsolve", [((15, 6, 5), 4400), ((5, 27, 5), 3500)], ids=str)
def test_euler_batches_of_many_planes(shape, nsolve):
    """3D grids on 2^a 3^b 5^c axes whose planes (first) or kept y modes
    (second) times solves pass 65535, the limit of two of a launch's three
    grid dimensions."""
    U0 = np.stack([euler_state(shape, i) for i in range(3)])

    def run(plan, U):
        f64 = dict(dtype=torch.float64, device="cuda")
        plan.run_(U, 2, 0.02 / max(shape))
        plan.run_cfl_(U, 2, torch.zeros(plan.nsolve, **f64), torch.full((plan.nsolve,), 1.0, **f64))
        return U

    same_alone(U0, nsolve, run, filter_params=FP, cfl=0.3)


@pytest.mark.parametrize("shape,nsolve", [((65, 3), 32300), ((3, 65), 32300)], ids=str)
@pytest.mark.parametrize("filt", [None, FP], ids=["plain", "filter"])
def test_lgl_batches_of_many_rows(shape, nsolve, filt):
    """Solves times rows of an LGL grid beyond 65535 tiles of 128."""
    r = np.random.RandomState(0)
    U0 = np.stack([euler_state(shape, i) for i in range(3)])
    U0[:, 1:3] *= 0.1 + 0.01 * r.standard_normal(shape)
    same_alone(U0, nsolve, lambda p, U: p.run_(U, 2, 1e-5), basis="legendre", filter_params=filt)


@pytest.mark.parametrize("shape,nsolve", [((8, 8), 65536), ((9, 8), 65536), ((8, 8, 8), 8192)], ids=str)
def test_batches_past_the_launch_limits_leave_the_state_alone(shape, nsolve):
    from phrike_gb300.engine import Plan
    U0 = torch.as_tensor(euler_state(shape, 0).astype(np.float32), device="cuda").expand(nsolve, -1, *shape).contiguous()
    plan = Plan(shape, (1.0,) * len(shape), nsolve=nsolve, filter_params=FP, cfl=0.3)
    f64 = dict(dtype=torch.float64, device="cuda")
    t, end = torch.zeros(nsolve, **f64), torch.full((nsolve,), 1.0, **f64)
    for run in (lambda U: plan.run_(U, 2, 1e-3), lambda U: plan.run_cfl_(U, 2, t, end)):
        U = U0.clone()
        with pytest.raises(RuntimeError):
            run(U)
        assert torch.equal(U, U0)
    assert float(t.abs().max()) == 0.0
