"""A context's first sweep, in which the buffers of the whole-GPU reduction grow from
one iteration to the next: the concurrent grids run side by side in it as they do
in the second sweep.  Where one grid's buffer was freed with the grid before it
running, the four ran one after the other (709 ms of Householder reductions
against 309); side by side they differ by little more than noise: 1.3."""
import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [tg.PREC_FP64, tg.PREC_MIXED], ids=["fp64", "mixed"])
def test_first_sweep_overlaps_its_grids(monkeypatch, precision):
    if precision == tg.PREC_MIXED:
        monkeypatch.setenv("NRG_MIXED_N", "2000")
    point = (2.5, 0.5606, -0.1902, 0.001758, 0.001758)
    warm = tg.Engine(0)
    warm.sweep("2chQS", 3, 60, *point, precision=precision)
    warm.close()
    e = tg.Engine(0)
    try:
        t = []
        for _ in range(2):
            e.sweep("2chQS", 5, 1500, *point, precision=precision)
            t.append(e.timing()["tridiag_ms"])
        assert t[0] < 1.3 * t[1]
    finally:
        e.close()
