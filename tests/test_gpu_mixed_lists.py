"""The mixed form with large blocks on both sides of its own threshold, dealt to
one and to four concurrent streams: every block is reduced once, by the FP64
whole-GPU kernel below the threshold and by the blocked panels from it on, also
where the call before left other block lists.  Levels within the mixed form's 1e-9
of the iteration's largest, integers exact."""
import os

import numpy as np
import pytest

import twochnrg_gb300 as tg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", ["1", "4"])
def test_both_kinds_of_large_blocks(engine, monkeypatch, split):
    from oracle import oracle as orc
    monkeypatch.setenv("NRG_BIG_N", "48")
    monkeypatch.setenv("NRG_MIXED_N", "150")
    monkeypatch.setenv("NRG_GRID_SPLIT", split)
    for kept in (200, 150):
        case = ("2chQS", 5, kept, 2.5, 0.3, -0.15, 0.01, 0.01)
        g = engine.sweep(*case, precision=tg.PREC_MIXED)
        o = orc.run(*case, nthreads=min(8, os.cpu_count() or 1))
        assert max(max(it.bsize) for it in g.iters) >= 150
        for a, b in zip(g.iters, o.iters):
            np.testing.assert_array_equal(a.bsize, b.bsize)
            np.testing.assert_array_equal(a.kept_bsize, b.kept_bsize)
            assert np.abs(a.en - b.en).max() < 1e-9 * max(1.0, np.abs(b.en).max())
