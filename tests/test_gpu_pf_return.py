"""mckl_b200_pf_ar1_plain_f64 returns with its work done: the final particles may
be read on another stream at once, whatever the number of steps (the particles
change buffers at every step)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [0, 1, 2, 3])
@pytest.mark.parametrize("N", [1000, 5000, 1 << 20])
def test_particles_are_final_on_return(N, T):
    require_cuda()
    import mckl_b200 as mb

    vp = ctypes.c_void_p
    y = np.linspace(0.0, 1.0, T + 1)
    key = (ctypes.c_uint32 * 2)(3, 4)
    ll = ctypes.c_double()
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.empty(N, dtype=torch.float64, device="cuda")
    W = torch.empty_like(x)
    z = torch.empty_like(x)
    args = (N, T, vp(y.ctypes.data), 0.9, 1.0, 0.5, 2.0, ctypes.cast(key, vp), ctypes.cast(key, vp), 2, 0.5,
            ctypes.byref(ll), None, None, None, vp(x.data_ptr()), vp(W.data_ptr()), vp(own.cuda_stream))
    torch.cuda.synchronize()
    for _ in range(10):
        assert mb._pf_plain(*args) == 0
        idle = own.query()
        with torch.cuda.stream(other):
            z.copy_(x)
        torch.cuda.synchronize()
        assert idle and torch.equal(x, z)
    # the same particles as from a run whose stream is read in order
    res = mb.pf_ar1_plain(N, y, 0.9, 1.0, 0.5, 2.0, (3, 4), (3, 4))
    assert torch.equal(res["x"], x) and torch.equal(res["W"], W)
