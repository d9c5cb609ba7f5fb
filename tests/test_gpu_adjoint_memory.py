"""The adjoint's working memory: an interval that the caller gives bounds it by the
header's formula; the default may keep the records of the whole run."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

F, N, T = 148, 4096, 100


def handle(mb):
    w = mb.batched_workload(F=F, T=T, seed=93, nmin=300, nmax=301)
    return mb.BatchedFilters(np.full(F, N), w["y"], w["phi"], w["sx"], w["sy"], w["mkeys"], w["rkeys"], fp64=True)


def used(call):
    """Device memory that `call` leaves taken."""
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    out = call()
    return before - torch.cuda.mem_get_info()[0], out


def formula(C):
    ctas = min(F, torch.cuda.get_device_properties(0).multi_processor_count)
    return 16 * F * N * (T // C + 1) + ctas * N * (C * 28 + 24)


SLACK = 32 << 20  # alignment, small arrays, the allocator's granularity, kernels loaded by the first call


def test_a_given_interval_bounds_the_memory():
    require_cuda()
    import mckl_b200 as mb

    b = handle(mb)
    out = []
    for C in (8, 32):
        n, r = used(lambda: b.adjoint(checkpoint_every=C))
        out.append(r)
        # the handle's buffer grows from the one to the other
        assert n <= formula(C) + SLACK, (C, n, formula(C))
    _, r = used(lambda: b.adjoint())
    out.append(r)
    b.close()
    for ll, g in out[1:]:
        assert np.array_equal(ll, out[0][0]) and np.array_equal(g, out[0][1])


def test_records_that_do_not_fit_leave_the_memory_alone():
    require_cuda()
    import mckl_b200 as mb

    b = handle(mb)
    want = b.adjoint(checkpoint_every=80)  # takes more than the default's checkpoints would
    # leave less than the whole run's records and more than nothing
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - formula(32), dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            n, (ll, g) = used(lambda: b.adjoint())
            assert n == 0, n
            assert np.array_equal(ll, want[0]) and np.array_equal(g, want[1])
    finally:
        del hold
        torch.cuda.empty_cache()
        b.close()
