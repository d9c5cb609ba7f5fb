"""A Gamma draw of one stream around the lengths where its CTA changes size (1024 values;
2048 with Threefry): bit for bit the block of gamma_blocks on the same counter, at a
shape of every algorithm and from an engine in the middle of a block."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

import oracle as O  # noqa: E402

ALPHA = np.array([0.3, 0.8, 1.0, 1.001, 2.5])


@pytest.mark.parametrize("kind", range(1, 7))
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_both_sides_of_the_line(kind, dt):
    require_cuda()
    import mckl_b200 as mb

    cls = list(mb.ENGINES.values())[kind - 1]
    orc = O.CPUPath("oracle")
    for n in (1, 511, 1023, 1024, 1025, 2047, 2048, 2049):
        g = cls()
        g.key = (5,)
        got = mb.gamma_blocks(g, n, ALPHA, dtype=dt).reshape(len(ALPHA), n)
        for b, a in enumerate(ALPHA):
            h = cls()
            h.key = (5,)
            _, key, tweak, index, _ = h.state_tuple()
            h.load_state([0, b, 0, 0], list(key), list(tweak), index)
            want = mb.gamma_distribution(h, n, alpha=float(a), dtype=dt)
            assert torch.equal(got[b].view(torch.uint8), want.view(torch.uint8)), (n, a)
        # the engine's state, from the middle of a block
        for a in (0.8, 2.5):
            e = O.Engine.make(kind, key=(5,), index=1)
            h = cls()
            h.load_state(list(e.ctr), list(e.key), list(e.tweak), e.index)
            orc.gamma(e, dt == "f64", n, a, 1.0)
            mb.gamma_distribution(h, n, alpha=a, dtype=dt)
            assert h.state_tuple() == e.state(), (n, a)
