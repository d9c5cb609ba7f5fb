"""Which batches have filters run by clusters of CTAs: the sizes that the tests of
the cluster step compare with the single CTA's take it, and the handles that give
the single CTA's results do not."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


def taken(N, shape=None, **kw):
    import mckl_b200 as mb

    F = len(N)
    w = mb.batched_workload(F=F, T=2, seed=5, nmin=300, nmax=301)
    b = mb.BatchedFilters(np.array(N), w["y"], w["phi"], w["sx"], w["sy"], w["mkeys"], w["rkeys"], **kw)
    if shape:
        b.config(*shape)
    n = b.cluster_filters()
    b.run()  # the count is of the launch that this makes
    b.results()
    b.close()
    return n


@pytest.mark.parametrize("N", [4097, 5119, 6851, 7168, 8191, 8192, 20001, 65536, 100003])
def test_one_large_filter(N):
    require_cuda()
    assert taken([N]) == 1
    assert taken([N], shadow=True) == 0 and taken([N], fp64=True) == 0
    assert taken([N] * 1301) == 0  # the batch fills the chip by itself


def test_mixed_batches():
    require_cuda()
    for shape in ((128, 8), (256, 1), (512, 2), (1024, 1)):
        assert taken([9001, 6851, 300, 30000], shape) == 3
    assert taken([7233, 6851, 4500]) == 3 and taken([4096, 300, 1]) == 0
    rng = np.random.default_rng(9)
    N = np.rint(np.exp(rng.uniform(np.log(256), np.log(40000), 400))).astype(int)
    assert taken(N) == int(np.sum(N > max(4096, N.sum() / (4 * torch.cuda.get_device_properties(0).multi_processor_count))))
