"""The grouped FP64 products with tiles of 8, 16 and 32 rows: the rows follow from
the number of tiles per SM, so a few states kept give the smallest tiles, some
hundreds the middle and some thousand the largest.  Averages against the oracle
and, for the backward sweep's products, the trace of rho; tolerances as in the
sweep tests."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", [5, 260, 500, 1000])
def test_rotations(engine, kept):
    args = ("1chQSz", 5, kept, 2.5, 0.4, -0.15, 0.02, 1e-3)
    g, o = engine.sweep(*args), orc.run(*args)
    for a, b in zip(g.iters, o.iters):
        assert a.nkept == b.nkept
        assert np.abs(a.en - b.en).max() < 1e-10 * np.abs(b.en).max()
        np.testing.assert_allclose(a.opavg, b.opavg, rtol=1e-8, atol=1e-12)


@pytest.mark.parametrize("kept", [5, 260, 600])
def test_density_matrices(engine, kept):
    engine.sweep_dm(8, kept, 2.5, 0.5, -0.2, 0.02)
    trace = engine.dm_backprop(engine.dm_params(temp=0.0))
    assert np.abs(trace - 1.0).max() < 1e-10
