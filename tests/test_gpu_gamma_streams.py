"""A stream of gamma_blocks and a Gamma draw of one stream are the same chunks at
two CTA sizes, all algorithms of a call in one launch: at lengths around a warp, a
CTA and a chunk, and at shapes of every algorithm (1.001: many redraws), block b has
to equal, bit for bit, the draw of an engine at counter (0, b), which
test_gpu_gamma holds against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

ALPHA = np.array([2.5, 0.3, 1.001, 1.0, 0.8, 1.2, 0.59, 40.0])


@pytest.mark.parametrize("engine", ["Philox4x32", "Threefry4x64_64", "ARS"])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_block_equals_single_stream(engine, dt):
    require_cuda()
    import mckl_b200 as mb

    K = 8192 // (4 if dt == "f32" else 8)
    for n in (1, 31, 33, 255, 257, K - 1, K, K + 1, 2 * K + 129, 5 * K + 3):
        g = mb.ENGINES[engine]()
        g.key = (3,)
        got = mb.gamma_blocks(g, n, ALPHA, dtype=dt).reshape(len(ALPHA), n)
        for b, a in enumerate(ALPHA):
            h = mb.ENGINES[engine]()
            h.key = (3,)
            _, key, tweak, index, _ = h.state_tuple()
            h.load_state([0, b, 0, 0], list(key), list(tweak), index)
            want = mb.gamma_distribution(h, n, alpha=float(a), dtype=dt)
            assert torch.equal(got[b].view(torch.uint8), want.view(torch.uint8)), (n, a)
