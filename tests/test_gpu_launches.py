"""The kernel launches that a flexible solve reports: those of its inner FP32
solves and of its FP64 applications, a split INT8 product's sum of parts among
them (over 2048 points along the reduction)."""
import numpy as np
import pytest

import fastmbcui_b200 as F
from fastmbcui_b200 import scenes as S
from fastmbcui_b200.flexible import solve_flexible

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _t(a, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")


@pytest.mark.parametrize("impl,per_apply", [("simt", 2), ("int8", 4)])
def test_flexible_solve_counts_its_launches(impl, per_apply):
    # per application: permute and one FP64 kernel, or permute, pack, MMA, sum
    sc = S.ellipsoids_scene(2, 1500, seed=21)
    plan = F.Plan(sc.y, sc.rho, sc.lam, sc.max_super)
    x, nx, y = _t(sc.x), _t(sc.nx), _t(sc.y)
    s64 = F.Solver(plan, x=x, nx=nx, y=y, coef=sc.coef, precision=F.MBC_F64).set_fp64_matvec(impl).prepare()
    s32 = F.Solver(plan, x=x, nx=nx, y=y, coef=sc.coef, precision=F.MBC_F32).factor()
    inner, solve = [], s32.solve_adjoint

    def counted(*a, **k):
        z, st = solve(*a, **k)
        inner.append(int(st["kernel_launches"]))
        return z, st

    s32.solve_adjoint = counted
    _, info = solve_flexible(s64, s32, _t(sc.rhs()), tol=1e-8, inner_iters=40)
    # fp64_applies counts K^T K products; one K^T more forms the right-hand side
    assert info["kernel_launches"] == sum(inner) + per_apply * (2 * info["fp64_applies"] + 1), (info, sum(inner))


def _kernels(f):
    """f's result and the kernels that ran on the device meanwhile."""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        r = f()
        torch.cuda.synchronize()
    dev = torch.autograd.DeviceType.CUDA
    return r, sum(e.device_type == dev and not e.name.startswith("Mem") for e in p.events())


@pytest.mark.parametrize("prec", [F.MBC_F64, F.MBC_F32])
@pytest.mark.parametrize("impl", ["simt", "int8"])
def test_counted_launches_are_those_that_ran(prec, impl):
    sc = S.ellipsoids_scene(2, 1500, seed=21)
    plan = F.Plan(sc.y, sc.rho, sc.lam, sc.max_super)
    s = F.Solver(plan, x=_t(sc.x), nx=_t(sc.nx), y=_t(sc.y), coef=sc.coef, precision=prec).set_fp64_matvec(impl)
    if impl == "int8":
        s.prepare()
    before = s.launches()
    _, ran = _kernels(s.factor)
    if ran == 0:
        pytest.skip("no device activity is recorded here")
    assert s.launches() - before == ran
    Fm = _t(sc.rhs(), torch.float64)
    for opts in ({}, {"schedule": F.MBC_SCHED_BLOCK}, {"fp64_recursion": 1}, {"true_residual": 1}):
        (_, st), ran = _kernels(lambda: s.solve(Fm, max_iters=400, **opts))
        assert st["kernel_launches"] == ran, opts


def test_first_use_check_of_the_int8_product_takes_the_split_path():
    # 3000 points: two parts.  Planes of two directions; the check's INT8 products
    # (pack, MMA, sum of parts, twice) and its FP64 products
    sc = S.ellipsoids_scene(2, 1500, seed=21)
    plan = F.Plan(sc.y, sc.rho, sc.lam, sc.max_super)
    s = F.Solver(plan, x=_t(sc.x), nx=_t(sc.nx), y=_t(sc.y), coef=sc.coef, precision=F.MBC_F64).set_fp64_matvec("int8")
    before = s.launches()
    s.prepare()
    assert s.launches() - before == 2 + 2 * 3 + 2
