"""The row kernel of the block tridiagonalization (k_rows.cu) through
nrg_diag_blocks, against numpy's eigh of the same blocks: at the edges of its
clusters (rows per CTA, CTAs without rows), strips and passes, on both sides of
the step where the dot product is split over the CTAs (193 rows) and of the
largest block it takes, with many blocks per cluster, and on blocks of
very large and very small scale.

Tolerances as in the other eigensolver tests, relative to the block's largest
level: eigenvalues 1e-12, residuals and orthogonality 1e-11.
"""
import numpy as np
import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu


def _block(n, seed, scale=1.0):
    rng = np.random.default_rng([n, seed])
    a = rng.standard_normal((n, n))
    return scale * (a + a.T)


def _check(engine, blocks):
    packed = np.concatenate([b[np.triu_indices(len(b))] for b in blocks])
    ev, vec = engine.diag_blocks([len(b) for b in blocks], packed)
    for b, w, z in zip(blocks, ev, vec):
        top = max(float(np.abs(np.linalg.eigvalsh(b)).max()), 1e-300)
        b, w = b / top, w / top
        assert np.abs(w - np.linalg.eigvalsh(b)).max() < 1e-12
        assert np.abs(b @ z.T - z.T * w).max() < 1e-11
        assert np.abs(z @ z.T - np.eye(len(b))).max() < 1e-11


@pytest.mark.parametrize("cluster", ["1", "2", "4", "8", "16"])
def test_edges(engine, monkeypatch, cluster):
    monkeypatch.setenv("NRG_ROWS_CLUSTER", cluster)
    _check(engine, [_block(n, 1) for n in (1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65, 127, 129)])


@pytest.mark.parametrize("n", [192, 193, 194, 195, 256, 321, 513, 616, 617, 618])
def test_sizes(engine, n):
    _check(engine, [_block(n, 2)])


def test_many_blocks_per_cluster(engine):
    # more blocks than clusters fit at once, one- and two-state blocks among them
    sizes = [90, 2, 1, 41, 3, 17, 2, 2, 5, 33] * 24
    _check(engine, [_block(n, k) for k, n in enumerate(sizes)])


@pytest.mark.parametrize("scale", [1e-40, 1e-25, 1e25])
def test_scaled_blocks(engine, scale):
    _check(engine, [_block(n, 3, scale) for n in (2, 3, 40, 200)])


@pytest.mark.parametrize("scale", [1e-140, 1e140])
def test_scales_refused_by_the_level_solver(engine, scale):
    # the level solver's FP32 bracket and inverse iteration end near 1e+-40
    b = _block(40, 3, scale)
    with pytest.raises(tg.NRGError):
        engine.diag_blocks([40], b[np.triu_indices(40)])


def test_blocks_that_fall_apart(engine):
    # zero columns (no reflector), a diagonal block, a zero block
    a = _block(50, 4)
    a[:25, 25:] = 0.0
    a[25:, :25] = 0.0
    _check(engine, [a, np.diag(np.arange(1.0, 21.0)), np.ones((30, 30))])
    ev, _ = engine.diag_blocks([12], np.zeros(78))
    assert np.array_equal(ev[0], np.zeros(12))
