"""What a caller sets decides which kernel a batch of few FP64-pair chains runs:
set_window(1) the one-step kernel with the tile's threads, and autotune() searches
on the kernel that will run."""
import numpy as np
import pytest

from mcgpu_gb300 import PREC_FP64, ROT_AXIS, ChainBatch, Context
from mcgpu_gb300.workloads import water_box

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def boxes(n, waters=130):
    return [water_box(waters + waters // 4 * (c % 6), cutoff=6.0, seed=c % 6) for c in range(n)]


def run(ctx, n_chains, window, steps=600, waters=130):
    bt = ChainBatch(ctx, boxes(n_chains, waters), list(range(n_chains)), rotation=ROT_AXIS)
    bt.set_precision(PREC_FP64)
    bt.set_tile(64, 1, 16)
    if window:
        bt.set_window(window)
    bt.run(steps)
    st, xyz = bt.stats()[:6], [np.stack(bt.download(c)) for c in range(6)]
    bt.close()
    return st, xyz


def test_window_of_one_is_the_one_step_kernel(ctx):
    """One and the same kernel adds a launch's energy changes in one order, so few
    chains with set_window(1) have the energies of the same chains among a hundred
    (which never run windows) to the last bit."""
    st, xyz = run(ctx, 6, 1)
    ref, rxyz = run(ctx, 100, 0)
    for a, b, x, y in zip(st, ref, xyz, rxyz):
        assert a.energy == b.energy and a.accepted == b.accepted
        assert np.array_equal(x, y)


def test_few_small_chains_run_one_step_at_a_time(ctx):
    """27 to 60 waters: most steps of a window would be evaluated twice."""
    st, xyz = run(ctx, 6, 0, waters=27)
    ref, rxyz = run(ctx, 100, 0, waters=27)
    for a, b, x, y in zip(st, ref, xyz, rxyz):
        assert a.energy == b.energy and a.accepted == b.accepted
        assert np.array_equal(x, y)


@pytest.mark.parametrize("window", [0, 1])
def test_autotune_searches_what_runs(ctx, window):
    """Unasked windows: only the steps of a launch; one step at a time: the tile."""
    bt = ChainBatch(ctx, boxes(6), list(range(6)), rotation=ROT_AXIS)
    bt.set_precision(PREC_FP64)
    bt.set_tile(32, 1, 7)
    if window:
        bt.set_window(window)
    before = np.stack(bt.download(3))
    threads, cpc, spl, lanes = bt.autotune(16)
    assert spl in (4, 16, 64)
    assert window or (threads, cpc, lanes) == (32, 1, 0)
    assert np.array_equal(before, np.stack(bt.download(3)))
    assert bt.stats()[3].steps == 0
    bt.close()
