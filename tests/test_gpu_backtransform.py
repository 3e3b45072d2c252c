"""The back-transformation by groups of reflectors and one reflector at a time
(k_tdeig.cu): sizes around a group of four, a warp's 32 columns and the size
where the second takes over, few and many vectors per block, against the
blocks themselves (residual and orthogonality 1e-11 of the largest level, as in
the other eigensolver tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[2, 3, 4, 5, 6, 7, 8, 9, 10, 11], [33, 34, 35, 36, 37, 66, 67], [300] * 5,
                                   [899, 40], [900], [901, 3, 120], [1743, 30]], ids=str)
def test_vectors(engine, sizes):
    rng = np.random.default_rng(sum(sizes))
    blocks = []
    for n in sizes:
        a = rng.standard_normal((n, n))
        blocks.append((a + a.T) / np.sqrt(n))
    ev, vec = engine.diag_blocks(sizes, np.concatenate([b[np.triu_indices(len(b))] for b in blocks]))
    for b, w, z in zip(blocks, ev, vec):
        top = np.abs(w).max()
        assert np.abs(b @ z.T - z.T * w).max() < 1e-11 * top
        assert np.abs(z @ z.T - np.eye(len(b))).max() < 1e-11
