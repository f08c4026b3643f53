"""Launches of many chains, whose groups take the chains in order for all their steps
(more than 128 chains per step of a segment), against the same chains among few, whose
groups choose by the work left: the same energies, counts and coordinates to the last
bit, with several chains per CTA, partial last segments and traces too."""
import numpy as np
import pytest

from mcgpu_gb300 import ROT_AXIS, ChainBatch, Context
from mcgpu_gb300.workloads import water_box
from test_gpu_fp64_items import CASES, mixed_box, one_primary

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def box(c):
    if c % 97 == 5:
        return one_primary(mixed_box(*CASES["uneven_edges"]))
    n = 5 + 11 * (c % 7)
    return water_box(n, seed=c % 7, cutoff=5.0, L=14.0)


@pytest.mark.parametrize("tile", [(64, 1), (256, 4)])
@pytest.mark.parametrize("steps", [2, 53, 150])
def test_many_equal_few(ctx, tile, steps):
    n, seg = 700, 2
    got = []
    for k in (n, 120):
        bt = ChainBatch(ctx, [box(c) for c in range(k)], list(range(k)), rotation=ROT_AXIS)
        bt.set_tile(tile[0], tile[1], seg)
        tr = bt.run_traced(steps)[:120] if steps == 53 else None
        if tr is None:
            bt.run(steps)
        assert all(s.steps == steps for s in bt.stats())
        got.append(([(s.energy, s.accepted, s.pairs) for s in bt.stats()[:120]],
                    [np.stack(bt.download(c)) for c in range(120)],
                    tr and [[(t.mol, t.accepted, t.de) for t in c] for c in tr]))
        bt.close()
    assert got[0][0] == got[1][0]
    assert all(np.array_equal(a, b) for a, b in zip(got[0][1], got[1][1]))
    assert got[0][2] == got[1][2]
