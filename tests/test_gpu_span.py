"""The span kernel (k_span.cu): one block by a group of CTAs of a cooperative
grid.  Routed to it by thresholds of 2 states: blocks smaller than the group,
around a strip of 32 columns and the 128 columns from which rows are split,
several blocks per group, rows left in L2; and by the rule itself, alone, beside
the row kernel and after the whole-GPU kernel.  Against the blocks themselves
(residual and orthogonality 1e-11 of the largest level, as in the other
eigensolver tests) and against the cluster kernel's levels (1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blocks(sizes, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n in sizes:
        a = rng.standard_normal((n, n)) * (0.6 / np.sqrt(n))
        a = a + a.T
        a[np.diag_indices(n)] += rng.uniform(0.0, 10.0, n)
        out.append(a)
    return out


def _diag(engine, blocks):
    return engine.diag_blocks([len(b) for b in blocks], np.concatenate([b[np.triu_indices(len(b))] for b in blocks]))


def _check(blocks, ev, vec):
    for b, w, z in zip(blocks, ev, vec):
        top = max(np.abs(w).max(), 1e-300)
        assert np.all(np.diff(w) >= 0)
        assert np.abs(b @ z.T - z.T * w).max() < 1e-11 * top
        assert np.abs(z @ z.T - np.eye(len(b))).max() < 1e-11


@pytest.mark.parametrize("sizes", [[3], [4, 3], [31, 32, 33, 34], [64, 127, 128, 129, 130, 131, 3, 5], [160] * 9,
                                   [257, 255, 100, 2, 1]], ids=str)
def test_small(engine, monkeypatch, sizes):
    monkeypatch.setenv("NRG_ROWS_N", "2")
    monkeypatch.setenv("NRG_SPAN_N", "2")
    blocks = _blocks(sizes, sum(sizes))
    ev, vec = _diag(engine, blocks)
    _check(blocks, ev, vec)
    monkeypatch.setenv("NRG_CLUSTER", "4")
    ref, _ = _diag(engine, blocks)
    for a, b in zip(ev, ref):
        assert np.abs(a - b).max() < 1e-12 * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("sizes", [[618], [700, 60, 451, 450, 449, 617], [1201, 640, 640, 640, 30], [1500, 900, 900, 20],
                                   [1801], [1900] * 3 + [650, 200]], ids=str)
def test_rule(engine, sizes):
    blocks = _blocks(sizes, sum(sizes))
    _check(blocks, *_diag(engine, blocks))


def test_special_blocks(engine):
    """A zero block, a diagonal one, one that splits after a few columns, and
    scales near the ends of the solver's range."""
    n = 640
    base = _blocks([n], 3)[0]
    split = base.copy()
    split[:40, 40:] = 0.0
    split[40:, :40] = 0.0
    blocks = [np.zeros((n, n)), np.diag(np.arange(n, dtype=float)), split, base * 1e30, base * 1e-30]
    _check(blocks, *_diag(engine, blocks))


def test_not_finite(engine):
    b = _blocks([640], 4)[0]
    for bad in (np.nan, np.inf):
        c = b.copy()
        c[5, 300] = c[300, 5] = bad
        with pytest.raises(Exception):
            _diag(engine, [c])
    _check([b], *_diag(engine, [b]))
