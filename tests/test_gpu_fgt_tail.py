"""The outermost tail of the Lehmann sums through moments (k_fgt.cu): frequencies
up to 27 widths past the last record, where the sums are down to 1e-290, against
the direct sums of the same records.

The direct sum's argument x is rounded to an ulp of t and x^2 to half an ulp,
27^2 of which are 1.6e-13 of a term; the moments' own error is a tenth of that:
4e-13 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bbroad", [0.3, 0.6])
def test_tail(engine, monkeypatch, bbroad):
    engine.sweep_dm(12, 90, 2.5, 0.5, -0.2, 0.02)
    prm = engine.dm_params(temp=1e-6, bbroad=bbroad)
    engine.dm_backprop(prm)
    rng = np.random.default_rng(4)
    base = np.linspace(0.0, 29.0 * bbroad, 120) + rng.uniform(0, 0.05, 120)
    # the first frequency moves the bins' edges against the records
    for shift in np.arange(8) / 64.0:
        om = np.exp(base + shift * bbroad)
        out = []
        for least in ("1", "1000000000"):
            monkeypatch.setenv("NRG_FGT_MIN", least)
            out.append(engine.lehmann(prm, omegas=np.concatenate([-om[::-1], om]))[1])
        a, b = out
        seen = np.abs(b) > 1e-290
        assert np.abs(b[seen]).min() < 1e-270  # the tail is reached
        assert np.all(np.abs(a - b)[seen] <= 4e-13 * np.abs(b)[seen])
