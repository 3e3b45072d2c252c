"""Shells loaded from snapshots whose energies do not start at 0: the range of keys
that the moments of the Gaussian lists cover (k_fgt.cu) follows the shell's own
energy range.  Against the direct sums of the same records, as test_gpu_fgt.py
(1e-11 relative)."""
import numpy as np
import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [-5.0, 0.5])
def test_shifted_energies(tmp_path, monkeypatch, shift):
    from oracle import oracle as orc
    ns = 8
    for N, s in enumerate(orc.dm_shells(ns, 80, 2.5, 0.4, -0.2, 0.015)):
        s["en"] = s["en"] + shift
        tg.write_dm_shell(str(tmp_path), "shifted", N, s)
    tg.write_code_pars(str(tmp_path), 2.5, ns, "shifted")
    om = np.concatenate([-np.logspace(0.5, -3, 60), np.logspace(-3, 0.5, 60)])
    e = tg.Engine(0)
    try:
        assert e.dm_load_bin(str(tmp_path), "shifted") == ns
        prm = e.dm_params(temp=0.5, bbroad=0.6)
        e.dm_backprop(prm)
        out = []
        for least in ("1", "1000000000"):
            monkeypatch.setenv("NRG_FGT_MIN", least)
            out.append(e.lehmann(prm, omegas=om)[1])
        assert np.all(np.isfinite(out[1])) and np.abs(out[1]).min() > 0.0
        assert np.all(np.abs(out[0] - out[1]) <= 1e-11 * np.abs(out[1]))
    finally:
        e.close()
