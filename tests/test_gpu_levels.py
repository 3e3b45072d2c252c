"""The level solver (k_tdeig.cu) on tridiagonals with known levels, through
nrg_diag_blocks: with 8, 4 and 1 lanes per level (the number of states in the
call decides), on blocks of 1 to a few hundred states, on blocks that split
into pieces and on levels that come in pairs split by round-off.

The solver stops at a few ulps of the spectral radius (8 in its bracket test),
and its Sturm counts have a backward error of a few more: 16 ulps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ULPS = 16 * np.finfo(float).eps


def _toeplitz(n):
    return 2 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)


def _levels(engine, blocks):
    packed = np.concatenate([b[np.triu_indices(len(b))] for b in blocks])
    return engine.diag_blocks([len(b) for b in blocks], packed)[0]


@pytest.mark.parametrize("sizes", [[1, 2, 3, 5, 31, 32, 33, 250], [100] * 24 + [32], [100] * 25, [97] * 50 + [14],
                                   [97] * 51], ids=["edges", "2432", "2500", "4864", "4947"])
def test_known_levels(engine, sizes):
    for n, w in zip(sizes, _levels(engine, [_toeplitz(n) for n in sizes])):
        k = np.arange(1, n + 1)
        exact = 4 * np.sin(k * np.pi / (2 * (n + 1))) ** 2
        assert np.abs(w - exact).max() <= ULPS * 4


@pytest.mark.parametrize("copies", [1, 40, 110], ids=["8 lanes", "4 lanes", "1 lane"])
def test_pairs_and_pieces(engine, copies):
    # Wilkinson's matrix: pairs of levels split far below the round-off; and a
    # tridiagonal that falls into pieces of 1 to 20 states
    wil = np.diag(np.abs(np.arange(-15.0, 16.0))) + np.eye(31, k=1) + np.eye(31, k=-1)
    rng = np.random.default_rng(5)
    e = rng.uniform(0.5, 1.0, 59)
    e[[0, 1, 5, 19, 39, 57]] = 0.0
    pieces = np.diag(rng.uniform(-3, 3, 60)) + np.diag(e, 1) + np.diag(e, -1)
    blocks = [wil, pieces] * copies
    ref = [np.linalg.eigvalsh(wil), np.linalg.eigvalsh(pieces)]
    for i, w in enumerate(_levels(engine, blocks)):
        r = ref[i % 2]
        assert np.abs(w - r).max() <= 2 * ULPS * np.abs(r).max()  # numpy's own error beside ours
