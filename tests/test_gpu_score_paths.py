"""The score kernel keeps a cloud of up to about 10 600 particles in shared
memory and a larger one in global memory, by the handle's largest filter.  The
same filter must give the same bits either way: alone in its handle, and beside
a filter too large for shared memory.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 33, 511, 4097, 10616])
def test_shared_and_global_clouds_agree(N):
    require_cuda()
    import mckl_b200 as mb

    w = mb.batched_workload(F=2, T=30, seed=81, nmin=300, nmax=301)

    def run(sizes):
        k = len(sizes)
        b = mb.BatchedFilters(np.array(sizes), w["y"][:k], w["phi"][:k], w["sx"][:k], w["sy"][:k], w["mkeys"][:k],
                              w["rkeys"][:k], fp64=True)
        b.config(512, 1)
        b.run()
        ll, nr = b.results()
        ls, g = b.score()
        b.close()
        return ll, nr, ls, g

    ll0, nr0, ls0, g0 = run([N])
    ll1, nr1, ls1, g1 = run([N, 10617])
    assert np.array_equal(ll0, ls0) and np.array_equal(ll1, ls1)
    assert nr0[0] == nr1[0] and ls0[0] == ls1[0]
    assert np.array_equal(g0[0], g1[0]) and np.all(np.isfinite(g0))
