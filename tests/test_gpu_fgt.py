"""The Lehmann sums through moments of key bins (k_fgt.cu) against the direct
sums of the same records (NRG_FGT_MIN forces either path): log-Gaussian and
Gaussian lists, even and uneven frequencies, one frequency, narrow and wide
broadening, frequencies far outside the band, and the tangents.

The dropped terms are below 3e-12 of a term at the end of the Gaussian's reach
and below 1e-15 of it within 18 widths; the rounding of either sum is a few
1e-14 of its terms: 1e-11 relative where the terms do not cancel, and for the
tangents, which do, 1e-11 of the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EVEN = np.concatenate([-np.logspace(0, -8, 40), np.logspace(-8, 0, 40)])
UNEVEN = np.sort(np.random.default_rng(3).uniform(-1, 1, 61))


def _both(engine, monkeypatch, call):
    out = []
    for least in ("1", "1000000000"):
        monkeypatch.setenv("NRG_FGT_MIN", least)
        out.append(call())
    return out


@pytest.mark.parametrize("temp", [1e-9, 3e-3])
@pytest.mark.parametrize("bbroad", [0.3, 0.6, 1.2])
@pytest.mark.parametrize("omegas", [EVEN, UNEVEN, np.array([1e-4]), np.array([2.0, 10.0, 60.0, -30.0])],
                         ids=["even", "uneven", "one", "far"])
def test_spectrum(engine, monkeypatch, temp, bbroad, omegas):
    engine.sweep_dm(14, 90, 2.5, 0.5, -0.2, 0.02)
    prm = engine.dm_params(temp=temp, bbroad=bbroad)
    engine.dm_backprop(prm)
    (_, a), (_, b) = _both(engine, monkeypatch, lambda: engine.lehmann(prm, omegas=omegas))
    assert np.all(np.abs(a - b) <= 1e-11 * np.abs(b))


@pytest.mark.parametrize("temp", [1e-9, 3e-3])
def test_tangents(engine, monkeypatch, temp):
    engine.grad_forward_dm(12, 60, 2.5, 0.5, -0.2, 0.02)
    prm = engine.dm_params(temp=temp, bbroad=0.6)
    engine.dm_backprop(prm)
    (_, a, da), (_, b, db) = _both(engine, monkeypatch, lambda: engine.lehmann_grad(prm, omegas=UNEVEN))
    assert np.all(np.abs(a - b) <= 1e-11 * np.abs(b))
    for x, y in zip(da, db):
        assert np.abs(x - y).max() <= 1e-11 * np.abs(y).max()
