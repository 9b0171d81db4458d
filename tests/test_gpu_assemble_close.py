"""FP32 collocation matrices where the normalized half-angle form cancels:
sources next to an edge or a vertex of a face (down to the resolution of FP32
coordinates), and faces with one distant vertex.  The bound is that of
test_gpu_assemble.py: one FP32 unit of the FP64 matrix, plus 1e-11 of the
largest entry for entries that cancel."""
import numpy as np
import pytest

from fastmbcui_b200 import mesh

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check(V, F, S):
    M64 = mesh.assemble(V, F, S, dtype=torch.float64).cpu().numpy()
    M32 = mesh.assemble(V, F, S).double().cpu().numpy()
    assert np.isfinite(M64).all() and np.isfinite(M32).all()
    assert np.all(np.abs(M32 - M64) <= 1.2e-7 * np.abs(M64) + 1e-11 * np.abs(M64).max())


def _mesh(rng, nf):
    V = rng.uniform(-1, 1, (3 * nf, 3)).astype(np.float32)
    return V, np.arange(3 * nf, dtype=np.int32).reshape(nf, 3)


@pytest.mark.parametrize("h", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("at", ["edge", "vertex"])
def test_sources_next_to_an_edge_or_a_vertex(h, at):
    rng = np.random.default_rng(8)
    V, F = _mesh(rng, 48)
    S = []
    for f in rng.integers(0, 48, 700):
        a, b, c = V[F[f]].astype(np.float64)
        t = rng.uniform(0.1, 0.9) if at == "edge" else 0.0
        p, e = a + t * (b - a), (b - a) / np.linalg.norm(b - a)
        out = p - c - e * ((p - c) @ e)  # away from the face, in its plane
        out /= np.linalg.norm(out)
        ang = rng.uniform(-0.4, 0.4)
        S.append(p + h * (np.cos(ang) * out + np.sin(ang) * np.cross(e, out)))
    _check(V, F, np.asarray(S, np.float32))


@pytest.mark.parametrize("far", [1e2, 1e4, 1e6, 1e8, 1e10, 1e13, 1e16])
def test_faces_with_a_distant_vertex(far):
    rng = np.random.default_rng(9)
    V, F = _mesh(rng, 40)
    V[F[::3, 1]] *= np.float32(far)
    _check(V, F, rng.uniform(-1.5, 1.5, (300, 3)).astype(np.float32))
