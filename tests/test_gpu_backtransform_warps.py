"""The back-transformation with two warps per vector beside short blocks, and one
warp on the same blocks where there are too many vectors for two: block lists
that follow the rule (blocks past 300 states, and the vectors counted by the
longest's length leave two sub-partitions each) on the device at hand, either
side of it.  Residuals and products of a block's vectors as in
test_gpu_backtransform_split.py (1e-11)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _two_warps(sizes):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return max(sizes) >= 300 and 2 * sum(n * n for n in sizes) <= 4 * sms * max(sizes)


def _largest_short(n):
    """The largest short block beside one of n states that still takes two warps."""
    k = 0
    while _two_warps([n, k + 1]):
        k += 1
    return k


@pytest.mark.parametrize("two", [True, False], ids=["two warps", "one warp"])
@pytest.mark.parametrize("n", [300, 301, 302])
def test_vectors(engine, n, two):
    short = _largest_short(n)
    if short < 3:
        pytest.skip("this device has too few SMs for two warps on every vector of such a block")
    sizes = [n, short, 1] if _two_warps([n, short, 1]) else [n, short - 1, 1]
    if not two:
        sizes = [n, short + 1, 2]
    assert _two_warps(sizes) == two
    rng = np.random.default_rng(n)
    blocks = []
    for m in sizes:
        a = rng.standard_normal((m, m))
        blocks.append((a + a.T) / np.sqrt(m))
    ev, vec = engine.diag_blocks(sizes, np.concatenate([b[np.triu_indices(len(b))] for b in blocks]))
    for b, w, z in zip(blocks, ev, vec):
        top = np.abs(w).max()
        assert np.abs(b @ z.T - z.T * w).max() < 1e-11 * top
        assert np.abs(z @ z.T - np.eye(len(b))).max() < 1e-11
