"""Fills of less than a block up to two blocks and one value, from a block's start: the
first values of one longer fill, and the engine where the longer calls leave it."""
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["Philox4x32", "Philox4x32_64", "Threefry4x64", "Threefry4x64_64", "ARS", "ARS_64"])
def test_tiny_fills(engine):
    require_cuda()
    import mckl_b200 as mb

    fills = [lambda g, k: mb.rand(g, k)]
    for t in ("f32", "f64"):
        fills.append(lambda g, k, t=t: mb.exponential_distribution(g, k, dtype=t))
        fills.append(lambda g, k, t=t: mb.u01_oc_distribution(g, k, dtype=t))
        fills.append(lambda g, k, t=t: mb.u01_canonical_distribution(g, k, dtype=t))
    for fill in fills:
        for n in range(1, 18):
            whole = mb.ENGINES[engine](key=(5, 6, 7, 8)[:2 if engine.startswith("Philox") else 4])
            part = whole.copy()
            want = fill(whole, 64)
            assert torch.equal(fill(part, n), want[:n]), (engine, n)
            assert torch.equal(fill(part, 20), want[n:n + 20]), (engine, n)
