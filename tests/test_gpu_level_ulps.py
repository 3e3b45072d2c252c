"""Levels of tridiagonals with 8, 4 and one lane per level (k_tdeig.cu): known
spectra, Wilkinson's pairs, blocks that fall into pieces, and two or three weakly
coupled copies of a piece, whose levels come in pairs and triples split by 1e-15
to 1e-12, against a bisection in long double.

The number of lanes follows from the rows of all blocks against the device's
lanes; the copies of each list are chosen so that every kernel takes its turn,
and the rule is asserted.  Bounds, in ulps of the spectral radius' bound: a level
stands alone within 8 (the bracket's end) and the counts' own error, 16; of a
pair or triple, 8 and 4 lanes end at a bracket of 19 and the counts' own error:
24; one lane accepts a resolved pair's step (16 and 8 from the counts) and a
group within 64: 24 and 72."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _rule(sizes):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    idle = 4.0 * sms * 32 * max(sizes) / sum(n * n for n in sizes)
    return 8 if idle >= 6 else 4 if idle >= 2 else 1, idle


def _copies(sizes, lanes):
    """As many copies of the list as take `lanes` lanes per level."""
    idle = _rule(sizes)[1]
    c = 1 if lanes == 8 else int(np.ceil(idle / (3.5 if lanes == 4 else 1.0)))
    assert _rule(sizes * c)[0] == lanes
    return c


def _levels(engine, blocks):
    packed = np.concatenate([b[np.triu_indices(len(b))] for b in blocks])
    return engine.diag_blocks([len(b) for b in blocks], packed)[0]


def _dense(d, e):
    return np.diag(d) + np.diag(e, 1) + np.diag(e, -1)


def _exact(d, e):
    d, e2 = d.astype(np.longdouble), e.astype(np.longdouble) ** 2
    r = np.abs(d).max() + 2 * np.sqrt(e2.max())
    lo, hi, k = np.full(len(d), -r), np.full(len(d), r), np.arange(len(d))
    for _ in range(66):
        x = (lo + hi) / 2
        q = d[0] - x
        c = (q < 0).astype(int)
        for i in range(1, len(d)):
            q = d[i] - x - e2[i - 1] / np.where(q == 0, np.longdouble(1e-300), q)
            c += q < 0
        lo, hi = np.where(c > k, lo, x), np.where(c > k, x, hi)
    return ((lo + hi) / 2).astype(float)


@pytest.mark.parametrize("lanes", [8, 4, 1])
def test_known(engine, lanes):
    ns = [1, 2, 3, 5, 31, 32, 33, 250]
    toep = [2 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1) for n in ns]
    ref = [4 * np.sin(np.arange(1, n + 1) * np.pi / (2 * (n + 1))) ** 2 for n in ns]
    toep.append(_dense(np.abs(np.arange(-15.0, 16.0)), np.ones(30)))
    ref.append(_exact(np.abs(np.arange(-15.0, 16.0)), np.ones(30)))
    rng = np.random.default_rng(5)
    d, e = rng.uniform(-3, 3, 60), rng.uniform(0.5, 1.0, 59)
    e[[0, 1, 5, 19, 39, 57]] = 0.0
    toep.append(_dense(d, e))
    ref.append(np.sort(np.concatenate([_exact(x, y) if len(x) > 1 else x for x, y in
                                       [(d[a:b], e[a:b - 1]) for a, b in
                                        zip([0, 1, 2, 6, 20, 40, 58], [1, 2, 6, 20, 40, 58, 60])]])))
    c = _copies([len(b) for b in toep], lanes)
    for i, w in enumerate(_levels(engine, toep * c)):
        b, r = toep[i % len(toep)], ref[i % len(toep)]
        assert np.abs(w - r).max() <= 16 * EPS * np.abs(b).sum(1).max()


@pytest.mark.parametrize("lanes", [8, 4, 1])
def test_pairs_and_triples(engine, lanes):
    rng = np.random.default_rng(17)
    blocks, ref, bound = [], [], []
    for m in (6, 12, 31):
        for split in (2e-15, 2e-14, 2e-13):
            d, e = rng.uniform(-1, 1, m), rng.uniform(0.2, 0.8, m - 1)
            for D, E, one in ((np.concatenate([d, d[::-1]]), np.concatenate([e, [split], e[::-1]]), 24),
                              (np.tile(d, 3), np.concatenate([e, [split], e, [0.7 * split], e]), 72)):
                blocks.append(_dense(D, E))
                ref.append(_exact(D, E))
                bound.append(one if lanes == 1 else 24)
    c = _copies([len(b) for b in blocks], lanes)
    for i, w in enumerate(_levels(engine, blocks * c)):
        i %= len(blocks)
        assert np.abs(w - ref[i]).max() <= bound[i] * EPS * np.abs(blocks[i]).sum(1).max(), (i, len(blocks[i]))
