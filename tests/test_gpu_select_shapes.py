"""In-place selection by its two kernels (one dimension, or two slots and four
dimensions at a time) around a whole grid of slots: bit for bit the gather by parent
index."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

GRID = 148 * 16 * 256  # threads of the largest grid


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("dim", [1, 2, 4, 5])
@pytest.mark.parametrize("N", [1, 257, GRID - 1, GRID, GRID + 1, 2 * GRID, 2 * GRID + 1])
def test_select_is_the_gather(N, dim, dtype):
    require_cuda()
    import mckl_b200 as mb

    rng = np.random.default_rng(N + dim)
    w = np.exp(rng.normal(0, 2, N))
    W = torch.from_numpy(w / w.sum()).cuda()
    idx = mb.rep_to_index(mb.resample(mb.Systematic, mb.Philox4x32(3), W), N)
    x = torch.from_numpy(rng.normal(size=(dim, N))).to(dtype).cuda()
    want = x[:, idx]
    mb.select(idx, x)
    assert torch.equal(x, want)
