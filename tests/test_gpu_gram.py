"""The Gram matrices of the supernodes up to 64 entries (gram_kernel) through
the factor they give, against the oracle: FP64 factors per column 1e-7, the
bound of the other factor tests; FP32 factors of well-conditioned scenes within
1e-3 of them (FP32 sums of up to 1500 rows, cancellation up to 1e3 kept out by
the pivot test).  Scenes with sets of all sizes, rows that end inside a panel,
few supernodes (rows cut into parts) and many."""
import numpy as np
import pytest

import oracle as O
import fastmbcui_b200 as F
from fastmbcui_b200 import scenes as S

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _t(a, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")


def _scene(pts, rho, seed):
    axes = (1.0, 0.8, 1.3)
    area = S.ellipsoid_area(axes, 200)
    sc = S.ellipsoid_fibonacci_scene(axes, pts, offset=0.7 * (area / pts) ** 0.5)
    sc.rho = rho
    return sc


@pytest.mark.parametrize("pts,rho", [(37, 2.0), (333, 3.0), (700, 4.5), (1500, 3.0), (1203, 6.0)])
@pytest.mark.parametrize("dense", [False, True])
def test_factor_matches_oracle(pts, rho, dense):
    sc = _scene(pts, rho, 1)
    pl = O.plan(sc.y, sc.rho, sc.lam, sc.max_super)
    plan = F.Plan(sc.y, sc.rho, sc.lam, sc.max_super)
    K = sc.dense_K().astype(np.float32)
    op = O.Op(sc.nf, sc.n, M=K.astype(np.float64)) if dense else O.Op.from_scene(sc)
    _, want, _ = O.factor(op, pl)
    kw = dict(M=_t(K)) if dense else dict(x=_t(sc.x), nx=_t(sc.nx), y=_t(sc.y), coef=sc.coef)
    lp = pl["lptr"]
    norm = lambda v: np.sqrt(np.add.reduceat(np.asarray(v) ** 2, lp[:-1]))
    got, _ = F.Solver(plan, precision=F.MBC_F64, **kw).factor().get_factor()
    assert np.all(norm(got - want) <= 1e-7 * norm(want))
    got, _ = F.Solver(plan, precision=F.MBC_F32, **kw).factor().get_factor()
    assert np.all(norm(got - want) <= 1e-3 * norm(want))
