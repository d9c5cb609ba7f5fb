"""The cooperative SMC kernels' error word (csrc/smc_coop.cu) outlives the growth of
the stream's working memory: what a call that does not synchronize left there is
reported once, by the stream's next call that does.  The word is set here from the
host; no kernel waits in vain."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


def test_error_word_survives_growth():
    require_cuda()
    import mckl_b200 as mb

    lib = mb.raw_lib()
    scratch = getattr(lib, "_ZN9mckl_b2007scratchEimP11CUstream_st")  # scratch(slot, bytes, stream)
    scratch.restype, scratch.argtypes = ctypes.c_void_p, [ctypes.c_int, ctypes.c_size_t, ctypes.c_void_p]
    stream = torch.cuda.Stream()
    vp = ctypes.c_void_p
    v = {n: torch.from_numpy(np.random.default_rng(n).normal(size=n)).cuda() for n in (3000, 1 << 20)}
    W = {n: torch.empty_like(x) for n, x in v.items()}
    torch.cuda.synchronize()
    ess = ctypes.c_double()

    def set_log(n, read):
        return lib.mckl_b200_weight_set_log(n, vp(W[n].data_ptr()), vp(v[n].data_ptr()),
                                            ctypes.byref(ess) if read else None, None, vp(stream.cuda_stream))

    lib.mckl_b200_weight_set_log.argtypes = [ctypes.c_size_t] + [vp] * 5
    assert set_log(3000, True) == 0

    class Word:  # the error word: the first of the results, slot 9
        __cuda_array_interface__ = {"shape": (1,), "typestr": "<i4", "version": 3,
                                    "data": (scratch(9, 16, stream.cuda_stream), False)}

    torch.cuda.synchronize()
    torch.as_tensor(Word(), device="cuda").fill_(1)
    torch.cuda.synchronize()
    assert set_log(1 << 20, False) == 0  # grows the working memory; does not read
    assert set_log(3000, True) == -4 and b"wait" in lib.mckl_b200_last_error()
    assert set_log(3000, True) == 0
    lib.mckl_b200_release_stream(vp(stream.cuda_stream))
