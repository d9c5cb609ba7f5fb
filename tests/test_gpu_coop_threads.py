"""Host threads that make different SMC calls on one stream at the same time: each
gets what it gets alone (the calls' exchange slots are separate)."""
import ctypes
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [5000, 30000])  # a cluster of tiles; tiles that exchange through global memory
def test_different_calls_on_one_stream(N):
    require_cuda()
    import mckl_b200 as mb

    vp = ctypes.c_void_p
    stream = torch.cuda.Stream()
    sp = vp(stream.cuda_stream)
    rng = np.random.default_rng(N)
    v = torch.from_numpy(rng.normal(size=N)).cuda()
    w = np.exp(rng.normal(0, 2, N))
    W = torch.from_numpy(w / w.sum()).cuda()
    rep0 = mb.resample(mb.Systematic, mb.Philox4x32(5), W)
    out = {k: torch.empty(N, dtype=t, device="cuda") for k, t in
           (("weight", torch.float64), ("resample", torch.int64), ("index", torch.int64), ("x", torch.float64),
            ("W", torch.float64))}
    y = np.array([0.0, 1.0, -0.5])
    key = (ctypes.c_uint32 * 2)(1, 2)
    ll = ctypes.c_double()

    def weight():
        return mb._weight_set_log(N, vp(out["weight"].data_ptr()), vp(v.data_ptr()), None, None, sp)

    def resample():
        return mb._resample(mb.Stratified, N, N, ctypes.byref(mb.Philox4x32(9).state), vp(W.data_ptr()),
                            vp(out["resample"].data_ptr()), sp)

    def index():
        return mb._rep_to_index(N, N, vp(rep0.data_ptr()), vp(out["index"].data_ptr()), sp)

    def particles():
        return mb._pf_plain(N, 2, vp(y.ctypes.data), 0.9, 1.0, 0.5, 2.0, ctypes.cast(key, vp), ctypes.cast(key, vp), 2,
                            0.5, ctypes.byref(ll), None, None, None, vp(out["x"].data_ptr()),
                            vp(out["W"].data_ptr()), sp)

    torch.cuda.synchronize()
    calls = {weight: ("weight",), resample: ("resample",), index: ("index",), particles: ("x", "W")}
    for call in calls:
        assert call() == 0
    torch.cuda.synchronize()
    want = {k: t.clone() for k, t in out.items()}
    wrong = []

    def work(call):
        for _ in range(200):
            if call() != 0:
                wrong.append(call.__name__)
            with torch.cuda.stream(stream):
                same = [torch.equal(out[k], want[k]) for k in calls[call]]
            if not all(same):
                wrong.append(call.__name__)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
