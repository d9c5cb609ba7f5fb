"""The cooperative SMC kernels (csrc/smc_coop.cuh) at the sizes where their
tiling changes: one tile (1024), a cluster of tiles (8 x 1024), one tile per SM
(148 x 1024), the tiles of 4096, 7168 and 8192 elements, and just past what the chip
holds (148 x 8192, the multi-kernel path); with the weights that send the exact
fold through its event loop, and genealogies whose copies come from far tiles.
Bars as in test_gpu_smc.py and test_gpu_pf.py: weights within 2 ULP, ESS within
1e-13, counts, parents and engine states identical.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

import oracle as O  # noqa: E402

EDGES = [1, 2, 1023, 1024, 1025, 2049, 8192, 8193, 148 * 1024, 148 * 1024 + 1, 148 * 4096 + 5, 148 * 7168, 148 * 8192,
         148 * 8192 + 1]


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
def test_weight_edges(env, N):
    mb, orc = env
    rng = np.random.default_rng(N)
    for sd in (0.5, 40.0):  # even weights; nearly all of them zero
        v = rng.normal(0, sd, N)
        W0, ess0 = orc.weight_set_log(v)
        w = mb.Weight(N)
        w.set_log(dev(v))
        assert ulps(w.data.cpu().numpy(), W0).max() <= 2
        assert abs(w.ess() - ess0) <= 1e-13 * ess0


def resample_and_index(mb, orc, scheme, W, M, key):
    g = mb.Philox4x32()
    g.key = key
    e = O.Engine.make(1, key=key)
    rep = mb.resample(scheme, g, dev(W), M)
    want = orc.resample(scheme, e, W, M)
    got = rep.cpu().numpy().astype(np.uint64)
    assert np.array_equal(got, want), (scheme, len(W), M, np.flatnonzero(got != want)[:5])
    assert g.state_tuple() == e.state()
    if M:
        idx = mb.rep_to_index(rep, M).cpu().numpy().astype(np.uint64)
        assert np.array_equal(idx, orc.rep_index(want, M)), (scheme, len(W), M)


@pytest.mark.parametrize("scheme", range(6))
@pytest.mark.parametrize("N", EDGES)
def test_resample_edges(env, scheme, N):
    mb, orc = env
    rng = np.random.default_rng(1000 * scheme + N)
    W = np.exp(rng.normal(0, 2, N))
    W /= np.cumsum(W)[-1]
    resample_and_index(mb, orc, scheme, W, N, (scheme + 1, 5))
    if N in (1025, 8193):
        resample_and_index(mb, orc, scheme, W, 3 * N, (scheme + 1, 6))
        resample_and_index(mb, orc, scheme, W, N // 3, (scheme + 1, 7))


@pytest.mark.parametrize("scheme", range(6))
@pytest.mark.parametrize("N", [1000, 7000, 30000, 400000, 1 << 20])
def test_resample_hard_weights(env, scheme, N):
    mb, orc = env
    rng = np.random.default_rng(N + scheme)
    cases = []
    one = np.zeros(N)
    one[N - 3] = 1.0  # every copy from one particle of the last tile
    cases.append(one)
    first = np.full(N, 1e-30)
    first[0] = 1.0
    cases.append(first)
    ties = np.full(N, 2.0**-55)  # 1/4 + 2^-55 ties: every element an event
    ties[0] = 0.25
    ties[N // 2:] = 1.5 / N
    cases.append(ties)
    lead = rng.random(N)
    lead[:3 * N // 4] = 0.0
    cases.append(lead / np.cumsum(lead)[-1])
    for k, W in enumerate(cases):
        resample_and_index(mb, orc, scheme, W, N, (k + 1, 9))


@pytest.mark.parametrize("scheme", range(6))
@pytest.mark.parametrize("N,threshold", [(1, 0.5), (3, 1.5), (1000, 0.5), (1024, 1.5), (1025, 0.5), (4999, 0.9),
                                         (8193, 0.5), (160001, 0.5)])
def test_filter_edges(env, scheme, N, threshold):
    mb, orc = env
    T = 12 if N < 100000 else 4
    sd0 = 1.0 / np.sqrt(1 - 0.9 * 0.9)
    _, y = orc.simulate_ar1(T, 0.9, 1.0, 0.5, sd0, (7, 0))
    y = np.array(y)
    y[3] += 9.0  # an outlier: the weights collapse onto a few particles
    want = orc.pf_ar1(N, y, 0.9, 1.0, 0.5, sd0, (11, 3), (12, 4), scheme, threshold)
    for record in (True, False):
        res = mb.pf_ar1_plain(N, y, 0.9, 1.0, 0.5, sd0, (11, 3), (12, 4), scheme=scheme, threshold=threshold,
                              record=record)
        assert np.array_equal(res["resampled"], want["resampled"])
        assert np.max(np.abs(res["ess"] - want["ess"]) / want["ess"]) <= 1e-12
        assert abs(res["loglik"] - want["loglik"]) <= 1e-10 * abs(want["loglik"])
        assert np.max(np.abs(res["x"].cpu().numpy() - want["x"])) <= 1e-12
        assert np.max(np.abs(res["W"].cpu().numpy() - want["W"])) <= 1e-13
    anc = mb.pf_ar1_plain(N, y, 0.9, 1.0, 0.5, sd0, (11, 3), (12, 4), scheme=scheme, threshold=threshold,
                          record=True)["anc"].cpu().numpy().astype(np.uint64)
    rows = want["resampled"] == 1
    assert np.array_equal(anc[rows], want["anc"][rows])
