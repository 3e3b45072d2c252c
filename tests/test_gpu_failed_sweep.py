"""A sweep that fails part of the way: the iterations before the failing one are
left as in a sweep that ends with them, their operator averages included, and so
are the DM-NRG shells.  The failure here is SetDegen's: a tolerance that holds
every level of an iteration makes it refuse more than 2048 of them."""
import ctypes

import numpy as np
import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu
ARGS = dict(ncutoff=700, lam=2.5, U=0.3, ed=-0.15)
EPS = 1e-14  # 2^53 times it holds every level


def _cfg(nsites):
    return tg.SweepConfig(tg.MODELS["1chQS"], nsites, ARGS["ncutoff"], ARGS["lam"], ARGS["U"], ARGS["ed"], 0.01, 0.0,
                          EPS, tg.PREC_FP64, 0.0)


@pytest.mark.parametrize("dm", [False, True], ids=["sweep", "dm"])
def test_results_before_the_failure(dm):
    e = tg.Engine(0)
    try:
        run = e.L.nrg_sweep_run_dm if dm else e.L.nrg_sweep_run
        assert run(e.h, ctypes.byref(_cfg(12))) == 5  # NRG_ERR_SIZE
        done = int(e.L.nrg_sweep_num_iterations(e.h))
        assert done > 2
        got = e._fetch(True)
        shells = int(e.L.nrg_dm_num_shells(e.h))
        assert shells == (done if dm else 0)
        assert run(e.h, ctypes.byref(_cfg(done))) == 0
        want = e._fetch(True)
        assert len(got.iters) == len(want.iters) == done
        for a, b in zip(got.iters, want.iters):
            np.testing.assert_array_equal(a.en, b.en)
            np.testing.assert_array_equal(a.thermo, b.thermo)
            np.testing.assert_array_equal(a.opavg, b.opavg)
            assert a.nkept == b.nkept and a.device_ms > 0.0
        assert run(e.h, ctypes.byref(_cfg(done + 1))) == 5
    finally:
        e.close()
