"""Dense-operator products (the mfs_torch operator's matrix) at the edges of
their tiles: 64 outputs, 64 positions, columns in units of 4 (FP32) and 8
(FP64), groups of 32, matrices cut over a cluster, and row strides and base
addresses that allow 16-, 8- or only 4-byte copies.

Tolerances: FP64 1e-12 and FP32 2e-5 relative, as for the other products.
"""
import numpy as np
import pytest

import fastmbcui_b200 as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nf,n,R,shift", [(3, 5, 1, 0), (64, 64, 4, 0), (65, 63, 6, 0), (320, 162, 6, 0),
                                          (130, 128, 9, 1), (257, 250, 17, 0), (513, 516, 18, 2), (640, 324, 31, 0),
                                          (300, 401, 33, 0), (1000, 2050, 48, 0), (20000, 700, 12, 0),
                                          (700, 20000, 28, 0)])
@pytest.mark.parametrize("prec", [F.MBC_F64, F.MBC_F32])
def test_products_match_dense(nf, n, R, shift, prec):
    g = torch.Generator(device="cuda").manual_seed(nf + R)
    buf = torch.randn(nf * n + shift, generator=g, device="cuda")
    M = buf[shift:].view(nf, n)  # shift floats past a 16-byte boundary
    dt, tol = (torch.float64, 1e-12) if prec == F.MBC_F64 else (torch.float32, 2e-5)
    V = torch.randn(n, R, generator=g, device="cuda", dtype=dt)
    W = torch.randn(nf, R, generator=g, device="cuda", dtype=dt)
    pts = np.random.default_rng(n).uniform(-1, 1, (n, 3)).astype(np.float32)
    s = F.Solver(F.Plan(pts), M=M, precision=prec)
    for got, want in ((s.apply_K(V), M.double() @ V.double()), (s.apply_KT(W), M.double().T @ W.double())):
        assert got.dtype == dt and got.shape == want.shape
        assert float(torch.linalg.norm(got.double() - want) / torch.linalg.norm(want)) <= tol
