"""NRG_ROWS_CLUSTER: the cluster sizes that exist are taken, anything else is the
default, and the levels are the same (1e-13 of the largest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", ["1", "2", "4", "8", "16", "0", "", "auto", "3", "-8", "32"])
def test_values(engine, monkeypatch, value):
    monkeypatch.setenv("NRG_ROWS_CLUSTER", value)
    rng = np.random.default_rng(8)
    sizes = [120, 40, 33, 32, 7, 2, 1]
    blocks = []
    for n in sizes:
        a = rng.standard_normal((n, n))
        blocks.append(a + a.T)
    ev, _ = engine.diag_blocks(sizes, np.concatenate([b[np.triu_indices(len(b))] for b in blocks]))
    for b, w in zip(blocks, ev):
        ref = np.linalg.eigvalsh(b)
        assert np.abs(w - ref).max() <= 1e-13 * np.abs(ref).max()
