"""SpectralSolver2D/3D.run advances in chunks of CFL steps on the device where
nothing has to look at single steps; on_step forces the loop that waits for
every step.  Both take the same steps (same dt rule, same pauses at outputs and
checkpoints), so times agree to the rounding of dt (the states' rounding: 1e-6
of a step) and states to the repository's 1e-5 of a field's norm."""
import numpy as np
import pytest

from test_gpu_truncated_spectra import check, euler_state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(64, 48), (32, 32), (16, 20, 24)]


def solver(shape, interval=1):
    from phrike_gb300 import equations, grid, solver as S
    fp = {"enabled": True, "p": 8, "alpha": 36.0, "interval": interval}
    if len(shape) == 2:
        g = grid.Grid2D(shape[1], shape[0], 1.0, 1.0, filter_params=fp)
        return S.SpectralSolver2D(g, equations.EulerEquations2D(gamma=1.4), cfl=0.3)
    g = grid.Grid3D(*reversed(shape), 1.0, 1.0, 1.0, filter_params=fp)
    return S.SpectralSolver3D(g, equations.EulerEquations3D(gamma=1.4), cfl=0.3)


@pytest.mark.parametrize("shape", SIZES, ids=str)
@pytest.mark.parametrize("interval", [1, 3])
@pytest.mark.parametrize("outputs", [0.3, 3.7, 100.0])
def test_chunks_equal_single_steps(shape, interval, outputs, tmp_path):
    U0 = euler_state(shape, 4).astype(np.float32)
    dt = solver(shape).compute_dt(U0)
    runs = []
    for step in (None, lambda *a: None):
        s = solver(shape, interval)
        out = tmp_path / str(step is None)
        out.mkdir(exist_ok=True)
        seen = []
        h = s.run(U0, 0.0, 9.4 * dt, output_interval=outputs * dt, checkpoint_interval=4.2 * dt, outdir=str(out),
                  on_output=lambda t, U: seen.append(t), on_step=step)
        runs.append((h, seen, s.U.double().cpu().numpy(), s.t, len(list(out.iterdir()))))
    (h0, seen0, U, t0, n0), (h1, seen1, V, t1, n1) = runs
    assert n0 == n1 and len(seen0) == len(seen1) and t0 == t1
    np.testing.assert_allclose(h0["time"], h1["time"], rtol=0, atol=1e-5 * dt)
    np.testing.assert_allclose(seen0, seen1, rtol=0, atol=1e-5 * dt)
    check(U, V, len(shape), False)


@pytest.mark.parametrize("change", ["state", "cfl", "dt"])
def test_what_the_host_changes_counts(change):
    """A callback that rescales the state, a CFL number set after construction
    and an overridden compute_dt act as in the loop of single steps."""
    shape = (32, 32)
    U0 = euler_state(shape, 4).astype(np.float32)
    dt = solver(shape).compute_dt(U0)
    runs = []
    for step in (None, lambda *a: None):
        s = solver(shape)
        if change == "cfl":
            s.cfl = 0.1
        if change == "dt":
            s.compute_dt = lambda U: 0.4 * dt

        def hook(t, U):
            if change == "state" and 0.0 < t < 5 * dt:
                U[3] *= 1.5
        h = s.run(U0, 0.0, 6.2 * dt, output_interval=2.5 * dt, on_output=hook, on_step=step)
        runs.append((h, s.U.double().cpu().numpy()))
    np.testing.assert_allclose(runs[0][0]["time"], runs[1][0]["time"], rtol=0, atol=1e-5 * dt)
    check(runs[0][1], runs[1][1], 2, False)
