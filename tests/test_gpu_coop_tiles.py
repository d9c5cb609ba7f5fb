"""The cooperative SMC kernels at the edges of every tile size (512 x 2 and 512 x 4
elements, 1024 x 3 to 1024 x 8, at most 148 tiles): the last cloud of one size and
the first of the next.  Bars as in test_gpu_coop.py.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

import oracle as O  # noqa: E402

EDGES = [148 * 1024 * k + d for k in range(1, 9) for d in (0, 1)]


@pytest.fixture(scope="module")
def env():
    require_cuda()
    import mckl_b200 as mb

    O.build()
    return mb, O.CPUPath("oracle")


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def ulps(a, b):
    d = np.abs(a - b)
    return np.where(d == 0, 0.0, d / np.spacing(np.maximum(np.abs(a), np.abs(b))))


@pytest.mark.parametrize("N", EDGES)
def test_weight_counts_and_parents(env, N):
    mb, orc = env
    rng = np.random.default_rng(N)
    v = rng.normal(0, 3.0, N)
    W0, ess0 = orc.weight_set_log(v)
    w = mb.Weight(N)
    w.set_log(dev(v))
    assert ulps(w.data.cpu().numpy(), W0).max() <= 2
    assert abs(w.ess() - ess0) <= 1e-13 * ess0
    for scheme in (0, 1, 2, 3):
        g = mb.Philox4x32()
        g.key = (scheme + 1, 5)
        e = O.Engine.make(1, key=(scheme + 1, 5))
        rep = mb.resample(scheme, g, dev(W0), N)
        want = orc.resample(scheme, e, W0, N)
        assert np.array_equal(rep.cpu().numpy().astype(np.uint64), want), scheme
        assert g.state_tuple() == e.state()
        idx = mb.rep_to_index(rep, N).cpu().numpy().astype(np.uint64)
        assert np.array_equal(idx, orc.rep_index(want, N)), scheme


@pytest.mark.parametrize("scheme", [0, 1, 2, 5])
@pytest.mark.parametrize("N", [148 * 2048, 148 * 2048 + 1, 148 * 3072 - 3, 148 * 5120 + 1, 148 * 6144])
def test_filter(env, scheme, N):
    mb, orc = env
    T = 3
    sd0 = 1.0 / np.sqrt(1 - 0.9 * 0.9)
    _, y = orc.simulate_ar1(T, 0.9, 1.0, 0.5, sd0, (7, 0))
    y = np.array(y)
    y[2] += 6.0
    want = orc.pf_ar1(N, y, 0.9, 1.0, 0.5, sd0, (11, 3), (12, 4), scheme, 0.9)
    res = mb.pf_ar1_plain(N, y, 0.9, 1.0, 0.5, sd0, (11, 3), (12, 4), scheme=scheme, threshold=0.9, record=True)
    assert np.array_equal(res["resampled"], want["resampled"]) and res["resampled"].sum() > 0
    assert np.max(np.abs(res["ess"] - want["ess"]) / want["ess"]) <= 1e-12
    assert abs(res["loglik"] - want["loglik"]) <= 1e-10 * abs(want["loglik"])
    assert np.max(np.abs(res["x"].cpu().numpy() - want["x"])) <= 1e-12
    rows = want["resampled"] == 1
    assert np.array_equal(res["anc"].cpu().numpy().astype(np.uint64)[rows], want["anc"][rows])
