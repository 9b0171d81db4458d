"""Dense operators whose rows are further apart than their columns (ldm > n,
which the C interface takes), with strides and base addresses that allow 16-, 8-
and 4-byte copies; what lies between the rows is NaN.  Tolerances as in
test_gpu_dense.py: FP64 1e-12 and FP32 2e-5 relative."""
import ctypes as C

import numpy as np
import pytest

import fastmbcui_b200 as F
from fastmbcui_b200 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nf,n,R", [(5, 3, 1), (130, 65, 9), (700, 1030, 18)])
@pytest.mark.parametrize("extra,shift", [(1, 0), (2, 0), (4, 0), (7, 1), (6, 2)])
@pytest.mark.parametrize("prec", [F.MBC_F64, F.MBC_F32])
def test_products(nf, n, R, extra, shift, prec):
    g = torch.Generator(device="cuda").manual_seed(nf + extra)
    ld = n + extra
    buf = torch.full((nf * ld + shift,), float("nan"), device="cuda")
    M = buf[shift:].view(nf, ld)[:, :n]
    M.copy_(torch.randn(nf, n, generator=g, device="cuda"))
    pts = np.random.default_rng(n).uniform(-1, 1, (n, 3)).astype(np.float32)
    s = F.Solver.__new__(F.Solver)  # the Python constructor makes M contiguous
    s.plan, s.precision, s.nf, s.n, s._stream, s._keep = F.Plan(pts), prec, nf, n, None, (buf,)
    op = _lib.Operator()
    op.kind, op.nf, op.n, op.M, op.ldm = _lib.MBC_OP_DENSE, nf, n, M.data_ptr(), ld
    h = C.c_void_p()
    _lib.check(F.load().mbc_solver_create(s.plan.handle, C.byref(op), prec, s._sp(), C.byref(h)), "create")
    s._h = h
    dt, tol = (torch.float64, 1e-12) if prec == F.MBC_F64 else (torch.float32, 2e-5)
    V = torch.randn(n, R, generator=g, device="cuda", dtype=dt)
    W = torch.randn(nf, R, generator=g, device="cuda", dtype=dt)
    for got, want in ((s.apply_K(V), M.double() @ V.double()), (s.apply_KT(W), M.double().T @ W.double())):
        assert float(torch.linalg.norm(got.double() - want) / torch.linalg.norm(want)) <= tol
