"""Large FP32 filters are run by a cluster of CTAs each when one CTA would be the
tail of the batch (csrc/pf_batched.cu: joint_filters).  The split keeps the
single CTA's arithmetic and order, so the log-likelihoods and resampling counts
must be the same bits.  The single CTA's are taken from handles with an FP64
shadow, which always run that way and whose FP32 part is the same step.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


def pair(mb, N, T, seed, shape=None, threshold=0.5, outlier=False):
    N = np.array(N)
    w = mb.batched_workload(F=len(N), T=T, seed=seed, nmin=300, nmax=301)
    if outlier:
        w["y"][:, T // 2] += 12.0  # the weights collapse: long runs of copies
    out = []
    for shadow in (False, True):
        b = mb.BatchedFilters(N, w["y"], w["phi"], w["sx"], w["sy"], w["mkeys"], w["rkeys"], threshold=threshold,
                              shadow=shadow)
        if shape:
            b.config(*shape)
        b.run()
        first = b.results()
        b.run(graph=True)
        again = b.results()
        assert np.array_equal(first[0], again[0]) and np.array_equal(first[1], again[1])
        out.append(first)
        b.close()
    return out


@pytest.fixture(scope="module")
def mb():
    require_cuda()
    import mckl_b200

    return mckl_b200


# one and two tiles per range, odd counts, partial chunks (many one-pair units),
# ranges past the end
@pytest.mark.parametrize("N", [4097, 5119, 6851, 7168, 8191, 8192, 20001, 65536, 100003])
@pytest.mark.parametrize("outlier", [False, True])
def test_cluster_equals_single_cta(mb, N, outlier):
    (l0, r0), (l1, r1) = pair(mb, [N], 24, 5, outlier=outlier)
    assert np.array_equal(l0, l1) and np.array_equal(r0, r1)
    assert r0[0] > 0


@pytest.mark.parametrize("shape", [(128, 8), (256, 1), (512, 2), (1024, 1)])
def test_cluster_equals_single_cta_at_every_shape(mb, shape):
    (l0, r0), (l1, r1) = pair(mb, [9001, 6851, 300, 30000], 16, 6, shape=shape)
    assert np.array_equal(l0, l1) and np.array_equal(r0, r1)


def test_mixed_batch(mb):
    rng = np.random.default_rng(9)
    N = np.rint(np.exp(rng.uniform(np.log(256), np.log(40000), 400))).astype(int)
    (l0, r0), (l1, r1) = pair(mb, N, 12, 7)
    assert np.array_equal(l0, l1) and np.array_equal(r0, r1)


def test_every_step_resamples(mb):
    (l0, r0), (l1, r1) = pair(mb, [7233, 6851, 4500], 12, 8, threshold=2.0)
    assert np.array_equal(l0, l1) and np.array_equal(r0, r1) and np.all(r0 == 12)
