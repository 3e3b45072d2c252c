"""The grouped FP64 products (gemm_tile.cuh) at block sizes around their 32-wide
tiles, 8-row warps and 16-deep chunks: operator rotations (the
one-channel models' averages against the oracle, which rotates with dgemm) and the backward sweep's
products (traces of rho, 1 at every shell).  Tolerances as in the sweep tests."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["1chQS", "1chQSz"])
@pytest.mark.parametrize("kept", [9, 33, 70, 131])
def test_rotations(engine, model, kept):
    args = (model, 5, kept, 2.5, 0.4, -0.15, 0.02, 1e-3)
    g, o = engine.sweep(*args), orc.run(*args)
    for a, b in zip(g.iters, o.iters):
        assert a.nkept == b.nkept
        assert np.abs(a.en - b.en).max() < 1e-10 * np.abs(b.en).max()
        np.testing.assert_allclose(a.opavg, b.opavg, rtol=1e-8, atol=1e-12)


@pytest.mark.parametrize("kept", [9, 33, 70, 131])
def test_density_matrices(engine, kept):
    engine.sweep_dm(10, kept, 2.5, 0.5, -0.2, 0.02)
    trace = engine.dm_backprop(engine.dm_params(temp=0.0))
    assert np.abs(trace - 1.0).max() < 1e-10
