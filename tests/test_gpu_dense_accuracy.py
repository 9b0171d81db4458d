"""Rounding error of the FP32 dense products against 64 bits: no larger than
that of 32 interleaved FP32 fused multiply-add chains per output added in a
tree (K) and of one chain per output (K^T), both emulated here.  The ratio of two such errors over at least 320 x 6 outputs
scatters by about 2 %; 4 % is allowed."""
import numpy as np
import pytest

import fastmbcui_b200 as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _lanes(A, B):
    """A B (m x k, k x r) as 32 FP32 chains per output, lane l taking positions
    l, l + 32, ..., then a tree over the lanes."""
    m, k = A.shape
    pad = -k % 32
    A = torch.nn.functional.pad(A, (0, pad)).double().view(m, -1, 32)
    B = torch.nn.functional.pad(B, (0, 0, 0, pad)).double().view(-1, 32, B.shape[1])
    acc = torch.zeros(m, 32, B.shape[2], device=A.device, dtype=torch.float64)
    for i in range(A.shape[1]):
        acc = torch.addcmul(acc, A[:, i, :, None], B[None, i]).float().double()
    while acc.shape[1] > 1:
        h = acc.shape[1] // 2
        acc = (acc[:, :h] + acc[:, h:]).float().double()
    return acc[:, 0]


def _chain(M, W):
    acc = torch.zeros(M.shape[1], W.shape[1], device=M.device, dtype=torch.float64)
    for i in range(M.shape[0]):
        acc = torch.addcmul(acc, M[i, :, None].double(), W[None, i].double()).float().double()
    return acc


@pytest.mark.parametrize("nf,n,R", [(320, 162, 6), (1280, 642, 48), (5120, 2562, 6), (30000, 3000, 12),
                                    (3000, 20000, 18), (513, 5000, 31), (2000, 60, 5), (320, 162, 32), (1280, 642, 28),
                                    (30000, 3000, 32), (640, 324, 9), (700, 1024, 4)])
@pytest.mark.parametrize("positive", [False, True])
def test_error_is_no_larger_than_that_of_chains(nf, n, R, positive):
    g = torch.Generator(device="cuda").manual_seed(nf + R)
    new = (lambda *s: torch.rand(*s, generator=g, device="cuda")) if positive else (
        lambda *s: torch.randn(*s, generator=g, device="cuda"))
    M, V, W = new(nf, n), new(n, R), new(nf, R)
    pts = np.random.default_rng(n).uniform(-1, 1, (n, 3)).astype(np.float32)
    s = F.Solver(F.Plan(pts), M=M, precision=F.MBC_F32)

    def error(got, want):
        return float(torch.linalg.norm(got.double() - want) / torch.linalg.norm(want))

    want = M.double() @ V.double()
    e, bound = error(s.apply_K(V), want), error(_lanes(M, V).float(), want)
    assert e <= 1.04 * bound, (e, bound)
    want = M.double().T @ W.double()
    e, bound = error(s.apply_KT(W), want), error(_chain(M, W).float(), want)
    assert e <= 1.04 * bound, (e, bound)

