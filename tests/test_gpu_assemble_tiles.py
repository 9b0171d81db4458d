"""FP32 collocation matrices at the edges of the kernel's tiles, 16 faces and
128 sources, and where a block walks several source tiles and ends short.
Tolerance as in test_gpu_assemble.py."""
import numpy as np
import pytest

from fastmbcui_b200 import mesh

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nf", [15, 16, 17])
@pytest.mark.parametrize("ns", [127, 128, 129])
def test_tile_edges(nf, ns):
    _check(nf, ns)


def test_blocks_of_several_source_tiles():
    _check(5003, 1157)  # 313 face tiles, 10 source tiles in blocks of 8 and 2


def _check(nf, ns):
    rng = np.random.default_rng(nf + ns)
    V = rng.uniform(-1, 1, (nf // 2 + 3, 3)).astype(np.float32)
    F = np.array([rng.choice(len(V), 3, replace=False) for _ in range(nf)]).astype(np.int32)
    S = rng.uniform(-1.5, 1.5, (ns, 3)).astype(np.float32)
    M64 = mesh.assemble(V, F, S, dtype=torch.float64).cpu().numpy()
    M32 = mesh.assemble(V, F, S).double().cpu().numpy()
    assert M32.shape == (nf, ns)
    assert np.all(np.abs(M32 - M64) <= 1.2e-7 * np.abs(M64) + 1e-11 * np.abs(M64).max())
