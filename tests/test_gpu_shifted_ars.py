"""ARS fills that start inside a block, around the length from which they take the
shifted shape (512 blocks per SM): the tail of one aligned fill."""
import pytest

torch = pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine,words", [("ARS", 4), ("ARS_64", 2)])
def test_both_sides_of_the_line(engine, words):
    require_cuda()
    import mckl_b200 as mb

    line = 512 * torch.cuda.get_device_properties(0).multi_processor_count * words
    fills = [lambda g, k: mb.rand(g, k), lambda g, k: mb.exponential_distribution(g, k, dtype="f32"),
             lambda g, k: mb.exponential_distribution(g, k, dtype="f64")]
    for n in (line - 1, line, line + 1, line + words + 1, 4 * line + 3):
        for off in range(1, words):
            for fill in fills:
                whole = mb.ENGINES[engine](key=(5, 6, 7, 8))
                part = whole.copy()
                part.discard(off)
                assert torch.equal(fill(part, n), fill(whole, n + words)[off:off + n]), (n, off)
