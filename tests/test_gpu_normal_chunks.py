"""Normal draws at the edges of the chunk kernel: one chunk and its last short
one, odd calls (whose last value comes from two words behind the chunk), the
line between the two CTA sizes (two chunks per SM), calls long enough for the
lists of pairs that miss the quick phases to be worked off, and an unaligned
start.  A long draw consumes the same words as one draw per chunk, which the
kernel for short calls makes, and has to give the same bits; the short draws are
held against the oracle (mean 0: double within 2 ULP of the value, single within
1e-6 of it)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

import oracle as O  # noqa: E402

NAMES = {1: "Philox4x32", 4: "Threefry4x64_64", 5: "ARS"}


def pair(mb, kind, index):
    e = O.Engine.make(kind, key=(5,), ctr=(2**32 - 40,), index=index)
    g = mb.ENGINES[NAMES[kind]]()
    g.load_state(list(e.ctr), list(e.key), list(e.tweak), e.index)
    return g, e


@pytest.mark.parametrize("kind", [1, 4, 5])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_normal_chunks(kind, dt):
    require_cuda()
    import mckl_b200 as mb

    orc = O.CPUPath("oracle")
    K = 8192 // (4 if dt == "f32" else 8)
    for n, sd, index in ((1, 0.5, None), (3, 1.0, 1), (K - 1, 1.0, None), (K, 2.0, 1), (K + 1, 1.0, None),
                         (2 * K + 1, 1.0, 1)):
        g, e = pair(mb, kind, index)
        want = orc.normal(e, dt == "f64", n, 0.0, sd).astype(np.float64)
        got = mb.normal_distribution(g, n, stddev=sd, dtype=dt).cpu().numpy().astype(np.float64)
        assert g.state_tuple() == e.state(), n
        tol = 2 * np.spacing(np.abs(want)) if dt == "f64" else 1e-6 * np.maximum(np.abs(want), 1e-30)
        assert np.all(np.abs(got - want) <= tol), (n, sd)


@pytest.mark.parametrize("kind", [1, 4, 5])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_long_draw_equals_draws_per_chunk(kind, dt):
    require_cuda()
    import mckl_b200 as mb

    K = 8192 // (4 if dt == "f32" else 8)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n, mean, sd, index in ((2 * sms * K, 0.0, 1.0, None), (2 * sms * K + 1, 0.0, 1.0, 1),
                               (16 * sms * K + 3 * K + 77, -1.0, 3.0, None)):
        g, _ = pair(mb, kind, index)
        got = mb.normal_distribution(g, n, mean=mean, stddev=sd, dtype=dt)
        g, _ = pair(mb, kind, index)
        want = torch.cat([mb.normal_distribution(g, min(K, n - i), mean=mean, stddev=sd, dtype=dt)
                          for i in range(0, n, K)])
        assert torch.equal(got.view(torch.uint8), want.view(torch.uint8)), (n, mean, sd)
