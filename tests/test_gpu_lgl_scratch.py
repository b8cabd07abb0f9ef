"""LGL plans that step by even and odd parts share buffers between the parts of
a step and with the right-hand side: the products with the flux derivatives (G),
the filter's states with the RK increments, the flux planes of rhs with the step
operands.  Whatever ran before on the plan, a call must give the same bits."""
import numpy as np
import pytest

from test_gpu_lgl_even_odd import state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nsolve", [(3, 3, 2), (4, 5, 3), (17, 16, 3), (24, 9, 2), (65, 40, 2), (129, 130, 1)])
@pytest.mark.parametrize("prec", ["fp32", "bf16x3"])
@pytest.mark.parametrize("filt,scheme", [(False, "rk4"), (True, "rk4"), (True, "rk2")])
def test_calls_do_not_depend_on_earlier_ones(nx, ny, nsolve, prec, filt, scheme):
    from oracle import lgl as L
    from phrike_gb300.engine import Plan
    ax, ay = L.LGLAxis(nx, 2.0), L.LGLAxis(ny, 2.0)
    U0 = torch.as_tensor(np.stack([state(ax, ay, i) for i in range(nsolve)]).astype(np.float32), device="cuda")
    kw = dict(basis="legendre", gemm_precision=prec, nsolve=nsolve, scheme=scheme,
              filter_params={"enabled": filt, "p": 8, "alpha": 36.0})
    f64 = dict(dtype=torch.float64, device="cuda")

    def cfl(p):
        U, t = U0.clone(), torch.zeros(nsolve, **f64)
        p.run_cfl_(U, 2, t, torch.as_tensor([1.0, 0.0, 1e-9][:nsolve], **f64))  # (one solve never starts)
        return U

    calls = [lambda p: p.step_(U0.clone(), 1e-5), lambda p: p.rhs(U0), lambda p: p.run_(U0.clone(), 3, 1e-5), cfl,
             lambda p: p.derivative(U0, 1)] + ([lambda p: p.filter(U0)] if filt else [])
    fresh = [call(Plan((ny, nx), (2.0, 2.0), **kw)) for call in calls]
    used = Plan((ny, nx), (2.0, 2.0), **kw)
    used.run_(U0 * 1e4, 2, 1e-5)
    for order in (range(len(calls)), reversed(range(len(calls)))):
        for i in order:
            assert torch.equal(calls[i](used), fresh[i]), i
    assert used.status() == 0


@pytest.mark.parametrize("prec,fields", [("fp32", 32), ("bf16x3", 32)])
def test_scratch_of_a_large_grid(prec, fields):
    """G (8 fields), increments (8), three bf16 parts of even and odd x and y
    operands (12) and the matrices: under 32 fields of a 513 x 513 batch."""
    from phrike_gb300.engine import Plan
    plan = Plan((513, 513), (2.0, 2.0), basis="legendre", gemm_precision=prec, nsolve=16,
                filter_params={"enabled": True, "p": 8, "alpha": 36.0})
    assert plan.scratch_bytes() < fields * 4 * 513 * 513 * 16
