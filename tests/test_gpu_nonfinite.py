"""NaN and infinities through the FP32 solver's products (3xTF32 on the tensor
cores from 8 columns on) and its tensor-core Gram matrices.

A source on a collocation point has the kernel value 0 / 0 = NaN.  It and a NaN
in the vector block, whatever its bits (arithmetic on the device returns
0x7fffffff, the host's is 0x7fc00000), reach exactly the rows and columns they
enter; the other entries are those of the product without them, bit for bit,
since every output is its own sum.  A factor whose sets hold a NaN fails."""
import numpy as np
import pytest

import oracle as O
import fastmbcui_b200 as F
from fastmbcui_b200._lib import MBC_NONSPD_PIVOT

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _t(a, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")


def _scene(nf, n, seed):
    rng = np.random.default_rng(seed)
    x, nx = (rng.uniform(-1.0, 1.0, (nf, 3)).astype(np.float32) for _ in range(2))
    y = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32) + np.float32(3.0)
    return x, nx, y


def _solver(x, nx, y):
    return F.Solver(F.Plan(y), x=_t(x), nx=_t(nx), y=_t(y), precision=F.MBC_F32)


@pytest.mark.parametrize("nf,n,R", [(300, 200, 1), (300, 200, 7), (300, 200, 8), (1000, 1100, 33), (3000, 2900, 130),
                                    (257, 513, 256)])
def test_coincident_point_gives_nan(nf, n, R):
    x, nx, y = _scene(nf, n, nf + R)
    i, j = nf // 3, n // 2
    rng = np.random.default_rng(R)
    V, W = _t(rng.standard_normal((n, R))), _t(rng.standard_normal((nf, R)))
    s = _solver(x, nx, y)
    want, want_t = s.apply_K(V), s.apply_KT(W)
    x[i] = y[j]
    s = _solver(x, nx, y)
    got, got_t = s.apply_K(V), s.apply_KT(W)
    rows, cols = np.arange(nf) != i, np.arange(n) != j
    assert torch.isnan(got[i]).all() and torch.equal(got[rows], want[rows])
    # row i of K enters every sum of K^T, so only NaN or not is compared
    assert torch.isnan(got_t[j]).all() and torch.isfinite(got_t[cols]).all() and torch.isfinite(want_t).all()


@pytest.mark.parametrize("bits", [0x7FFFFFFF, 0xFFFFFFFF, 0x7FC00000, 0x7F800001, 0xFFC01000])
@pytest.mark.parametrize("R", [3, 12, 100])
def test_nan_of_any_bits_stays_in_its_column(bits, R):
    x, nx, y = _scene(500, 400, 3)
    s = _solver(x, nx, y)
    rng = np.random.default_rng(1)
    for apply, rows in ((s.apply_K, 400), (s.apply_KT, 500)):
        V = _t(rng.standard_normal((rows, R)))
        want = apply(V)
        V.view(torch.int32)[17, R // 2] = bits - (1 << 32) if bits >> 31 else bits
        got = apply(V)
        keep = np.arange(R) != R // 2
        assert torch.isnan(got[:, R // 2]).all() and torch.equal(got[:, keep], want[:, keep])


@pytest.mark.parametrize("value", [float("inf"), float("-inf")])
def test_infinite_entry_is_not_lost(value):
    x, nx, y = _scene(500, 400, 4)
    s = _solver(x, nx, y)
    V = _t(np.random.default_rng(2).standard_normal((400, 16)))
    want = s.apply_K(V)
    V[5, 3] = value
    got = s.apply_K(V)
    keep = np.arange(16) != 3
    assert not torch.isfinite(got[:, 3]).any() and torch.equal(got[:, keep], want[:, keep])


@pytest.mark.parametrize("dense", [False, True])
def test_nan_in_a_tensor_core_gram_fails_the_factor(dense):
    # One body whose point j is only in sets of 64 to 150 entries, all of them
    # formed on the tensor cores; the points lie close to the collocation
    # points, so that no pivot of the sound factor asks for the FP64 retry.
    k = np.arange(150) + 0.5
    z, phi = 1.0 - k / 75.0, np.pi * (1.0 + 5.0 ** 0.5) * k
    nx = np.stack([np.sqrt(1.0 - z * z) * np.cos(phi), np.sqrt(1.0 - z * z) * np.sin(phi), z], 1).astype(np.float32)
    x, y = nx.copy(), (np.float32(0.97) * nx).astype(np.float32)
    pl = O.plan(y, 60.0, 1.5, 2048)
    smallest = np.full(150, 1 << 30)
    for a, b in zip(pl["set_ptr"][:-1], pl["set_ptr"][1:]):
        smallest[pl["set_ind"][a:b]] = np.minimum(smallest[pl["set_ind"][a:b]], b - a)
    j = int(pl["Pinv"][np.flatnonzero(smallest >= 64)[0]])  # in the original order
    plan = F.Plan(y, 60.0, 1.5, 2048)
    r = x[:, None, :].astype(np.float64) - y[None]
    K = (np.einsum("ijk,ik->ij", r, nx.astype(np.float64)) / np.linalg.norm(r, axis=2) ** 3).astype(np.float32)

    def solver():
        kw = dict(M=_t(K)) if dense else dict(x=_t(x), nx=_t(nx), y=_t(y))
        return F.Solver(plan, precision=F.MBC_F32, **kw)

    s = solver().factor()
    assert s.tensor_grams() > 0 and s.pivot_retries() == 0
    if dense:
        K.view(np.int32)[40, j] = 0x7FFFFFFF
    else:
        x[40] = y[j]
    with pytest.raises(F.MbcError) as e:
        solver().factor()
    assert e.value.status == MBC_NONSPD_PIVOT
