"""FP64 point-kernel products (K, K^T, the single-layer potential) at the edges
of their tiles: 16 outputs, 64 staged positions, 8-column tiles, column
groups of 96, and the split reductions of mid sizes.

Tolerance 1e-12 relative per product, the FP64 kernels' (test_gpu_parity.py):
sums of up to 5000 terms of one sign-mixed kernel, each to a few ulps.
"""
import numpy as np
import pytest

import oracle as O
import fastmbcui_b200 as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _points(rng, m):
    return rng.uniform(-1.0, 1.0, (m, 3)).astype(np.float32)


def _t(a, dt):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")


@pytest.mark.parametrize("nf,n,R", [(1, 5, 1), (15, 17, 8), (16, 64, 9), (65, 63, 1), (129, 200, 25), (803, 801, 6),
                                    (777, 1030, 41), (300, 333, 96), (130, 260, 97), (500, 450, 192),
                                    (5000, 4999, 3), (4500, 5000, 60)])
def test_products_match_oracle(nf, n, R):
    rng = np.random.default_rng(nf * 31 + R)
    x, nx = _points(rng, nf), _points(rng, nf)
    y = _points(rng, n) + np.float32(3.0) * (rng.integers(0, 2, (n, 1)) * 2 - 1).astype(np.float32)
    V, W = rng.standard_normal((n, R)), rng.standard_normal((nf, R))
    op = O.Op(nf, n, x=x, nx=nx, y=y, coef=-0.25)
    s = F.Solver(F.Plan(y), x=_t(x, torch.float32), nx=_t(nx, torch.float32), y=_t(y, torch.float32), coef=-0.25)
    for got, want in ((s.apply_K(_t(V, torch.float64)), op.K(V)), (s.apply_KT(_t(W, torch.float64)), op.KT(W))):
        got = got.cpu().numpy()
        assert got.shape == want.shape
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


def test_nan_column_stays_in_its_column():
    rng = np.random.default_rng(5)
    x, nx, y = _points(rng, 100), _points(rng, 100), _points(rng, 90) + np.float32(4.0)
    s = F.Solver(F.Plan(y), x=_t(x, torch.float32), nx=_t(nx, torch.float32), y=_t(y, torch.float32))
    V = _t(rng.standard_normal((90, 10)), torch.float64)
    want = s.apply_K(V)
    V[7, 3] = float("nan")
    V[8, 5] = float("inf")
    got = s.apply_K(V)
    keep = [c for c in range(10) if c not in (3, 5)]
    assert torch.equal(got[:, keep], want[:, keep])
    assert torch.isnan(got[:, 3]).all() and not torch.isfinite(got[:, 5]).any()
