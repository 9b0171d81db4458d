"""The one-column-at-a-time schedule with right-hand side and solution of
different types, and an odd number of rows: the FP64 column lies behind an odd
number of FP32 values in the schedule's buffer.  Against the batched solve: the
same PCG per column, so the same solution to 1e-6 of its norm at tol 1e-10 (the
fitted scenes' conditioning is below 1e3)."""
import numpy as np
import pytest

import fastmbcui_b200 as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rhs", [torch.float32, torch.float64])
@pytest.mark.parametrize("out", [torch.float32, torch.float64])
@pytest.mark.parametrize("start", [False, True])
def test_types_and_odd_sizes(rhs, out, start):
    nf, n = 501, 203
    g = torch.Generator(device="cuda").manual_seed(1)
    M = torch.randn(nf, n, generator=g, device="cuda")
    b = torch.randn(nf, 3, generator=g, device="cuda", dtype=torch.float64).to(rhs)
    pts = np.random.default_rng(0).uniform(-1, 1, (n, 3)).astype(np.float32)
    s = F.Solver(F.Plan(pts), M=M, precision=F.MBC_F64).factor()
    kw = dict(out_dtype=out, tol=1e-10, max_iters=500)
    X0 = torch.zeros(n, 3, device="cuda", dtype=out) if start else None
    want, _ = s.solve(b, X0=X0, **kw)
    got, st = s.solve(b, X0=X0, schedule=F.MBC_SCHED_PER_RHS, **kw)
    assert st["n_converged"] == 3 and got.dtype == out
    assert float(torch.linalg.norm((got - want).double()) / torch.linalg.norm(want.double())) <= 1e-6
    adj, st = s.solve_adjoint(want.to(rhs), schedule=F.MBC_SCHED_PER_RHS, **kw)
    ref, _ = s.solve_adjoint(want.to(rhs), **kw)
    assert st["n_converged"] == 3
    assert float(torch.linalg.norm((adj - ref).double()) / torch.linalg.norm(ref.double())) <= 1e-6
