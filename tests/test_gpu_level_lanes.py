"""The level solver with 8, 4 and one lane per level (k_tdeig.cu): the rule goes by
the blocks' rows per level against the GPU's lanes, so the same size alone, some
and many times over takes each; and one long block among many short ones.  Levels
against numpy (1e-12 of the largest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[300] * 8, [300] * 11, [300] * 16, [300] * 32, [300] * 40, [500] + [20] * 300,
                                   [1] * 5000 + [2] * 40], ids=lambda s: f"{s[0]}x{len(s)}")
def test_levels(engine, sizes):
    rng = np.random.default_rng(len(sizes))
    blocks = []
    for n in sizes:
        a = rng.standard_normal((n, n)) / np.sqrt(n)
        blocks.append(a + a.T)
    ev, _ = engine.diag_blocks(sizes, np.concatenate([b[np.triu_indices(len(b))] for b in blocks]))
    for b, w in zip(blocks, ev):
        ref = np.linalg.eigvalsh(b)
        assert np.abs(w - ref).max() < 1e-12 * np.abs(ref).max()
