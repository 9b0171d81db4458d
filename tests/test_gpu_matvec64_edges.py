"""FP64 point-kernel products at the kernel's own edges: 64 outputs a block, 64
staged positions, column groups of at most 64; and points at any finite
coordinates.  Tolerance as in test_gpu_matvec64.py: 1e-12 relative."""
import numpy as np
import pytest

import oracle as O
import fastmbcui_b200 as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _t(a, dt):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")


def _case(nf, n, R):
    rng = np.random.default_rng(nf * 31 + R)
    x, nx = (rng.uniform(-1.0, 1.0, (nf, 3)).astype(np.float32) for _ in range(2))
    y = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    y += np.float32(3.0) * (rng.integers(0, 2, (n, 1)) * 2 - 1).astype(np.float32)
    return x, nx, y, rng.standard_normal((n, R)), rng.standard_normal((nf, R))


def _solver(x, nx, y):
    return F.Solver(F.Plan(y), x=_t(x, torch.float32), nx=_t(nx, torch.float32), y=_t(y, torch.float32), coef=-0.25)


@pytest.mark.parametrize("nf,n", [(63, 65), (64, 64), (65, 63), (1000, 1001)])
@pytest.mark.parametrize("R", [63, 64, 65, 128, 129])
def test_products_match_oracle(nf, n, R):
    x, nx, y, V, W = _case(nf, n, R)
    op = O.Op(nf, n, x=x, nx=nx, y=y, coef=-0.25)
    s = _solver(x, nx, y)
    for got, want in ((s.apply_K(_t(V, torch.float64)), op.K(V)), (s.apply_KT(_t(W, torch.float64)), op.KT(W))):
        got = got.cpu().numpy()
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("scale", [1e12, 1e15, 1e18])
def test_point_far_away_stays_finite(scale):
    x, nx, y, V, W = _case(100, 90, 5)
    x[17] = scale  # (not the sources: the plan orders them by distance)
    s = _solver(x, nx, y)
    op = O.Op(100, 90, x=x, nx=nx, y=y, coef=-0.25)
    for got, want in ((s.apply_K(_t(V, torch.float64)), op.K(V)), (s.apply_KT(_t(W, torch.float64)), op.KT(W))):
        got = got.cpu().numpy()
        assert np.isfinite(got).all() and np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
