"""FP32 collocation matrices whose meshes have a vertex with a coordinate that
is NaN, infinite or far away (1e20, a parked vertex): only the faces that name
it are affected, wherever they stand among the 16 faces of a tile and whatever
the order of the tile's faces.  The bound is the one of test_gpu_assemble.py
for the other faces: one FP32 unit of the FP64 matrix, plus 1e-11 of the
largest entry."""
import numpy as np
import pytest

from fastmbcui_b200 import mesh

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf"), 1e20, -3e38])
@pytest.mark.parametrize("where", [0, 5, 16, 39])
def test_outlying_vertex_changes_only_its_faces(bad, where):
    rng = np.random.default_rng(int(where))
    V = rng.uniform(-1, 1, (60, 3)).astype(np.float32)
    F = np.array([rng.choice(59, 3, replace=False) for _ in range(40)]).astype(np.int32)
    F[where, 0] = 59  # the only face that names vertex 59
    S = rng.uniform(-1.5, 1.5, (150, 3)).astype(np.float32)
    want = mesh.assemble(V, F, S).cpu().numpy()
    V[59, 1] = bad
    M64 = mesh.assemble(V, F, S, dtype=torch.float64).cpu().numpy()
    M32 = mesh.assemble(V, F, S).double().cpu().numpy()
    assert np.array_equal(np.isnan(M64), np.isnan(M32))
    other = np.arange(40) != where
    assert np.isfinite(M32[other]).all()
    assert np.abs(M32[other] - want[other]).max() <= 1.2e-7 * np.abs(want[other]).max()
    ok = ~np.isnan(M64)
    assert np.all(np.abs(M32 - M64)[ok] <= 1.2e-7 * np.abs(M64[ok]) + 1e-11 * np.abs(M64[other]).max())


def test_outlying_source_changes_only_its_column():
    rng = np.random.default_rng(4)
    V = rng.uniform(-1, 1, (30, 3)).astype(np.float32)
    F = np.array([rng.choice(30, 3, replace=False) for _ in range(33)]).astype(np.int32)
    S = rng.uniform(-1.5, 1.5, (140, 3)).astype(np.float32)
    want = mesh.assemble(V, F, S).cpu().numpy()
    S[7, 0], S[129, 2] = float("nan"), float("inf")
    M64 = mesh.assemble(V, F, S, dtype=torch.float64).cpu().numpy()
    got = mesh.assemble(V, F, S).cpu().numpy()
    assert np.array_equal(np.isnan(M64), np.isnan(got))
    other = ~np.isin(np.arange(140), (7, 129))
    assert np.abs(got[:, other] - want[:, other]).max() <= 1.2e-7 * np.abs(want[:, other]).max()
