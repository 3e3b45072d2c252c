"""Device memory of the DM-NRG shells when one sweep follows another on a context:
no more than a fresh context needs, though the shells take over the memory of
those before, and nothing of the earlier sweep after one that fails."""
import ctypes

import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu
POINT = (2.5, 0.3, -0.15, 0.01)


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info(0)
    return total - free


def _pass(e, nsites, kept):
    e.sweep_dm(nsites, kept, *POINT)
    prm = e.dm_params(temp=1e-4, bbroad=0.6)
    e.dm_backprop(prm)


def test_shells_of_growing_sweeps():
    _pass(tg.Engine(0), 4, 60)  # what the process itself holds
    base = _used()
    a = tg.Engine(0)
    _pass(a, 16, 1000)
    fresh = _used() - base
    a.close()
    base = _used()
    b = tg.Engine(0)
    for kept in (960, 980, 1000):
        _pass(b, 16, kept)
    again = _used() - base
    b.close()
    assert again < 1.15 * fresh  # the context's own buffers grow by halves, as ever


def test_failed_sweep_frees_the_shells_before():
    e = tg.Engine(0)
    _pass(e, 24, 640)
    full = _used()
    cfg = tg.SweepConfig(tg.MODELS["1chQS"], 24, 640, *POINT, 0.0, 1e-14, tg.PREC_FP64, 0.0)
    assert e.L.nrg_sweep_run_dm(e.h, ctypes.byref(cfg)) == 5  # SetDegen refuses the first large iteration
    left = int(e.L.nrg_dm_num_shells(e.h))
    assert left < 8
    # 24 - left shells of at least 2000 states in 34 blocks, eigenvectors and rho
    assert full - _used() > (24 - left) * 2 * 8 * 2000 ** 2 // 34
    e.close()
