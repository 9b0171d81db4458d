"""The mixed-precision solve after residual replacements whose true residual
lies above the recursive one: the columns start their direction over and
converge in about the FP64 iterations, instead of carrying a stale direction.

Bound: each FP32 cycle gains at least the replacement factor 1e-2, so 1e-10
takes at most five cycles, each no longer than the FP64 solve to its own
1e-10 and rounded up to check_every: 5 (iterations of FP64 + 8)."""
import numpy as np
import pytest

import fastmbcui_b200 as F
from fastmbcui_b200 import scenes as S

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _t(a, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")


@pytest.mark.parametrize("axes,pts", [((0.6, 0.9, 1.3), 211), ((1.4, 0.7, 1.0), 737), ((1.5, 1.5, 0.5), 803)])
def test_mixed_iterations_follow_fp64(axes, pts):
    # sources about a point spacing inside
    area = S.ellipsoid_area(axes, 200)
    sc = S.ellipsoid_fibonacci_scene(axes, pts, offset=1.15 * (area / pts) ** 0.5)
    plan = F.Plan(sc.y, sc.rho, sc.lam, sc.max_super)
    pt = dict(x=_t(sc.x), nx=_t(sc.nx), y=_t(sc.y), coef=sc.coef)
    s64 = F.Solver(plan, precision=F.MBC_F64, **pt).factor()
    _, st64 = s64.solve(_t(sc.rhs(), torch.float64), tol=1e-10, max_iters=2000)
    s32 = F.Solver(plan, precision=F.MBC_F32, **pt).factor()
    _, st = s32.solve(_t(sc.rhs()), out_dtype=torch.float64, tol=1e-10, max_iters=2000)
    assert st["n_converged"] == 6 and st["true_relres_max"] <= 1e-10, st
    assert st["iters_max"] <= 5 * (st64["iters_max"] + 8), (st, st64["iters_max"])
