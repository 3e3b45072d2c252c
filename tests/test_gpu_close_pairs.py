"""Eigenvectors of blocks whose levels come in pairs split by 1e-16 to 1e-13 of the
spectral radius, as the channel doublets of the two-channel model do: inverse
iteration leaves two vectors of a pair at any angle to each other, and what
Gram-Schmidt makes of nearly parallel ones must not be round-off.

A vector's residual is a few ulps of the spectral radius, at most twenty times
that where a twentieth of it remains after the projection: 64 ulps.  Products of different
vectors are bounded by the ulps over the smallest gap that is not orthogonalized
(1e-4 of the radius), 2e-12, and a factor of a few: 1e-11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _block(n, rng):
    lam = rng.uniform(0, 16, n)
    h = n // 2
    lam[h:2 * h] = lam[:h] + 16 * 10.0 ** rng.uniform(-16, -13, h)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    a = (q * lam) @ q.T
    return 0.5 * (a + a.T)


@pytest.mark.parametrize("sizes", [[300] * 24 + [2, 3, 5, 33, 34], [901], [4] * 300], ids=["many", "901", "small"])
def test_vectors(engine, sizes):
    rng = np.random.default_rng(len(sizes))
    blocks = [_block(n, rng) for n in sizes]
    ev, vec = engine.diag_blocks(sizes, np.concatenate([b[np.triu_indices(len(b))] for b in blocks]))
    for b, w, z in zip(blocks, ev, vec):
        top = np.abs(w).max()
        assert np.abs(z @ b - w[:, None] * z).max() < 64 * np.finfo(float).eps * top
        assert np.abs(z @ z.T - np.eye(len(b))).max() < 1e-11
