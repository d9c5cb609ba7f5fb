"""The adjoint keeps the records of a whole run when they take no more than 4 GiB
and otherwise replays blocks from checkpoints.  Both must give the same bits: the
same filters in a handle large enough for checkpoints (148 x 8192 particles x 130
steps is just above the limit) and in smaller handles, at several checkpoint
intervals, T below, at and above the interval.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


def grads(mb, w, F, N, every):
    b = mb.BatchedFilters(np.full(F, N), w["y"][:F], w["phi"][:F], w["sx"][:F], w["sy"][:F], w["mkeys"][:F],
                          w["rkeys"][:F], fp64=True)
    b.config(1024, 1)
    out = [b.adjoint(checkpoint_every=e) for e in every]
    b.run()
    ll, _ = b.results()
    b.close()
    for l, g in out[1:]:
        assert np.array_equal(l, out[0][0]) and np.array_equal(g, out[0][1])
    assert np.array_equal(ll, out[0][0])
    return out[0]


def test_whole_records_equal_checkpoints():
    require_cuda()
    import mckl_b200 as mb

    w = mb.batched_workload(F=148, T=130, seed=91, nmin=300, nmax=301)
    l0, g0 = grads(mb, w, 148, 8192, (16, 50))
    l1, g1 = grads(mb, w, 3, 8192, (1, 16, 129, 130, 500))
    assert np.array_equal(l0[:3], l1) and np.array_equal(g0[:3], g1)
    assert np.all(np.isfinite(g0))


@pytest.mark.parametrize("N,T", [(1, 1), (7, 2), (1025, 3)])
def test_shortest_runs(N, T):
    require_cuda()
    import mckl_b200 as mb

    w = mb.batched_workload(F=2, T=T, seed=92, nmin=300, nmax=301)
    _, g = grads(mb, w, 2, N, (1, 2, 64))
    assert np.all(np.isfinite(g))
