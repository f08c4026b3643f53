"""ChainStats.pairs of chains with FP64 pairs: the atom pairs their steps evaluated,
which is what the same chains count with FP32 pairs (the same moves, in-range sets and
decisions), one step at a time, in windows, with lists and without."""
import pytest

from mcgpu_gb300 import PREC_FP64, PREC_MIXED, ROT_AXIS, ChainBatch, Context
from mcgpu_gb300.workloads import water_box
from test_gpu_fp64_items import CASES, mixed_box, one_primary

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("skin", [0.0, 1.0])
@pytest.mark.parametrize("window", [1, 4])
def test_fp64_chains_count_their_pairs(ctx, window, skin):
    boxes = [water_box(300, cutoff=7.0, seed=1), water_box(512, cutoff=9.0, seed=2),
             one_primary(mixed_box(*CASES["lengths_1_to_64"]))]
    got = []
    for prec in (PREC_FP64, PREC_MIXED):
        bt = ChainBatch(ctx, boxes, [4, 5, 6], rotation=ROT_AXIS)
        bt.set_precision(prec)
        bt.set_tile(128, 1, 16)
        bt.set_window(window)
        if skin:
            bt.set_verlet(skin)
        bt.run(160)
        got.append([(s.accepted, s.pairs) for s in bt.stats()])
        bt.close()
    assert got[0] == got[1]
    assert all(p > 0 for _, p in got[0])
