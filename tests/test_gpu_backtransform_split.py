"""The back-transformation with two warps per vector (few vectors of blocks of 300
states or more): the smallest such block, odd sizes, a vector whose partner in
the CTA is missing, and beside short blocks.  Kept states of a sweep against the
oracle's spectrum as in the sweep tests, and blocks' own residuals (1e-11)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[300], [301, 3], [299], [303, 2, 1, 5], [302, 40]], ids=str)
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


def test_sweep(engine):
    """Few kept vectors of blocks past 300 states: the next iteration's levels
    follow from them."""
    from oracle import oracle as orc
    args = ("2chQS", 4, 200, 2.5, 0.3, -0.15, 0.01, 0.01)
    g, o = engine.sweep(*args), orc.run(*args, nthreads=8)
    assert max(max(it.bsize) for it in g.iters) >= 300
    for a, b in zip(g.iters, o.iters):
        assert a.nkept == b.nkept
        assert np.abs(a.en - b.en).max() < 1e-10 * np.abs(b.en).max()
