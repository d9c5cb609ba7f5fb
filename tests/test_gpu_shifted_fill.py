"""Fills that start inside a block (the shifted shape of csrc/rng.cu, from 4096
values on): every engine, one-word transform and offset, at sizes around the
warps' 31 groups and the last partial group.  The words before the offset are
skipped by drawing them, so the values must equal the tail of one aligned fill.
"""
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["Philox4x32", "Philox4x32_64", "Threefry4x64", "Threefry4x64_64", "ARS", "ARS_64"])
@pytest.mark.parametrize("n", [4095, 4096, 4097, 31 * 8 * 32 + 5, 100003])
def test_offset_fill_is_the_tail_of_an_aligned_one(engine, n):
    require_cuda()
    import mckl_b200 as mb

    fills = [lambda g, k: mb.rand(g, k)]
    for t in ("f32", "f64"):
        fills.append(lambda g, k, t=t: mb.exponential_distribution(g, k, lam=1.5, dtype=t))
        fills.append(lambda g, k, t=t: mb.u01_oo_distribution(g, k, dtype=t))
        fills.append(lambda g, k, t=t: mb.u01_cc_distribution(g, k, dtype=t))
    for fill in fills:
        for off in range(1, 8):
            whole = mb.ENGINES[engine](key=(5, 6, 7, 8)[:2 if engine.startswith("Philox") else 4])
            part = whole.copy()
            part.discard(off)
            want = fill(whole, n + 8)[off:off + n]
            got = fill(part, n)
            assert torch.equal(got, want), (engine, n, off)
