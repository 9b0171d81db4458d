"""FP32 collocation matrices at the edges of their tiles (32 faces, 64
sources), with faces that share no vertex, sources on, next to and far from
faces, and coordinates of very small and very large scale.

Tolerance: every entry within one FP32 unit (1.2e-7 relative, half a unit of
rounding and its tie) of the FP64 matrix, plus 1e-11 of the largest entry for
entries that cancel."""
import numpy as np
import pytest

from fastmbcui_b200 import mesh

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check(V, F, S):
    M64 = mesh.assemble(V, F, S, dtype=torch.float64).cpu().numpy()
    M32 = mesh.assemble(V, F, S).double().cpu().numpy()
    assert np.array_equal(np.isnan(M64), np.isnan(M32))
    ok = ~np.isnan(M64)
    assert np.all(np.abs(M32 - M64)[ok] <= 1.2e-7 * np.abs(M64[ok]) + 1e-11 * np.abs(M64[ok]).max())
    return M64


@pytest.mark.parametrize("nf,ns,shared,scale", [(1, 1, False, 1.0), (31, 63, False, 1.0), (32, 64, True, 1.0),
                                                (33, 65, True, 1.0), (320, 162, True, 1e-3), (257, 1000, False, 1e4),
                                                (70, 130, True, 1e-25), (70, 130, False, 1e18)])
def test_fp32_matrix_matches_fp64(nf, ns, shared, scale):
    rng = np.random.default_rng(nf + ns)
    nv = max(3, nf // 2 + 2) if shared else 3 * nf
    V = (scale * rng.uniform(-1, 1, (nv, 3))).astype(np.float32)
    F = (np.array([rng.choice(nv, 3, replace=False) for _ in range(nf)]) if shared
         else np.arange(3 * nf).reshape(nf, 3)).astype(np.int32)
    S = (scale * rng.uniform(-1.5, 1.5, (ns, 3))).astype(np.float32)
    S[: ns // 4] = V[F[rng.integers(0, nf, ns // 4)]].mean(1)  # in a face
    S[ns // 4: ns // 3] *= np.float32(20.0)                      # far away
    _check(V, F, S)


def test_invalid_vertices_and_source_on_a_vertex():
    rng = np.random.default_rng(2)
    V = rng.uniform(-1, 1, (20, 3)).astype(np.float32)
    F = np.array([rng.choice(20, 3, replace=False) for _ in range(40)]).astype(np.int32)
    F[0, 0], F[7, 2], F[33, 1] = 20, -1, 1 << 30
    S = np.concatenate([V[:5], rng.uniform(-1, 1, (70, 3)).astype(np.float32)])
    M64 = _check(V, F, S)
    assert np.isnan(M64[[0, 7, 33]]).all()
