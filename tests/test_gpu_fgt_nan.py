"""A weight that is not finite (an infinite or NaN element of a loaded c_d) in the
Lehmann sums through moments (k_fgt.cu): every frequency that the direct sums
spoil is spoilt, however far its records are, and no other."""
import numpy as np
import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, np.nan, 1e200])
def test_spoilt_frequencies(tmp_path, monkeypatch, value):
    from oracle import oracle as orc
    ns = 8
    for N, s in enumerate(orc.dm_shells(ns, 80, 2.5, 0.4, -0.2, 0.015)):
        if N == 4:
            el = np.array(s["cd_el"])
            el[np.argmax(np.abs(el))] = value
            s["cd_el"] = el
        tg.write_dm_shell(str(tmp_path), "spoilt", N, s)
    tg.write_code_pars(str(tmp_path), 2.5, ns, "spoilt")
    om = np.concatenate([-np.logspace(6, -6, 80), np.logspace(-6, 6, 80)])
    e = tg.Engine(0)
    try:
        assert e.dm_load_bin(str(tmp_path), "spoilt") == ns
        prm = e.dm_params(temp=1e-3, bbroad=0.3)
        e.dm_backprop(prm)
        out = []
        for least in ("1", "1000000000"):
            monkeypatch.setenv("NRG_FGT_MIN", least)
            out.append(e.lehmann(prm, omegas=om)[1])
        spoilt = ~np.isfinite(out[1])
        assert spoilt.any()
        np.testing.assert_array_equal(~np.isfinite(out[0]), spoilt)
    finally:
        e.close()
