"""Log-weights of minus infinity in the batched FP32 filters: a filter run by a
cluster of CTAs gives what one CTA gives, so its result does not depend on the
other filters of the batch.  One observation overflows the FP32 likelihood of
every particle, or (sy tiny, so that only the particles near it have a finite
one) of some.  The single CTA's results are those of a handle with an FP64 shadow.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


def run(mb, N, y, sy, shadow):
    F = len(N)
    w = mb.batched_workload(F=F, T=y.shape[0] - 1, seed=31, nmin=300, nmax=301)
    b = mb.BatchedFilters(np.array(N), np.tile(y, (F, 1)), np.full(F, 0.9), np.ones(F), np.full(F, sy), w["mkeys"],
                          w["rkeys"], shadow=shadow)
    b.run()
    out = b.results()
    b.close()
    return out


@pytest.mark.parametrize("N", [4097, 6851, 20001, 65536])
@pytest.mark.parametrize("sy,at", [(0.5, 1e30), (1e-18, 25.0), (1e-18, 28.0), (0.5, np.inf)])
@pytest.mark.parametrize("first", [False, True])
def test_cluster_equals_single_cta(N, sy, at, first):
    require_cuda()
    import mckl_b200 as mb

    y = np.full(9, 0.3)
    y[1 if first else 5] = at
    l0, r0 = run(mb, [N], y, sy, False)
    l1, r1 = run(mb, [N], y, sy, True)
    np.testing.assert_array_equal(l0, l1)
    assert np.array_equal(r0, r1)
    # the same filter in a batch that fills the chip by itself, where none is joint
    lb, rb = run(mb, [N] + [N] * 1300, y, sy, False)
    np.testing.assert_array_equal(lb[:1], l0)
    assert rb[0] == r0[0]
