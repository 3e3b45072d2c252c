"""A wait of the span kernel that runs out (the limit set to one clock, so that the
first poll that finds an entry empty gives up): the call ends with its own status,
not with what the void numbers lead to, and the context goes on."""
import numpy as np
import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu


def _run(engine, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = a + a.T
    ev, _ = engine.diag_blocks([n], a[np.triu_indices(n)])
    return a, ev[0]


@pytest.mark.parametrize("n", [640, 1000])
def test_wait_runs_out(engine, monkeypatch, n):
    monkeypatch.setenv("NRG_SPAN_WAIT", "1")
    with pytest.raises(tg.NRGError) as e:
        _run(engine, n)
    assert e.value.status == 7  # NRG_ERR_TIMEOUT
    monkeypatch.delenv("NRG_SPAN_WAIT")
    a, w = _run(engine, n)
    ref = np.linalg.eigvalsh(a)
    assert np.abs(w - ref).max() < 1e-12 * np.abs(ref).max()
