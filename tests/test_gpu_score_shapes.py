"""score()'s log-likelihoods are run()'s on the same handle bit for bit, whatever
block shape the handle has: the filter's step runs on the handle's threads inside
the score kernel's larger CTAs.  Clouds in shared memory and past it, odd sizes,
and an outlier that collapses the weights."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [None, (128, 8), (256, 1), (512, 2), (1024, 1)])
@pytest.mark.parametrize("sizes", [(1, 33, 257, 2000, 4999), (9682, 300), (9683, 301), (10616, 77), (10617, 5003)])
def test_score_is_the_handles_run(shape, sizes):
    require_cuda()
    import mckl_b200 as mb

    k = len(sizes)
    w = mb.batched_workload(F=k, T=20, seed=94, nmin=300, nmax=301)
    w["y"][:, 11] += 9.0
    b = mb.BatchedFilters(np.array(sizes), w["y"], w["phi"], w["sx"], w["sy"], w["mkeys"], w["rkeys"], fp64=True)
    if shape:
        b.config(*shape)
    b.run()
    ll, nr = b.results()
    ls, g = b.score()
    _, nrs = b.results()
    b.close()
    assert np.array_equal(ls, ll) and np.array_equal(nrs, nr)
    assert np.all(np.isfinite(g))
