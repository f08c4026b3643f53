"""A chain's FP64 system energy is the same, bit for bit, alone and among any other
chains of a batch: its sum must not follow from where the chain lies in the pool or
how many molecules the pool has (a CTA sums up to eight molecules of a large box)."""
import pytest

from mcgpu_gb300 import ROT_AXIS, ChainBatch, Context
from mcgpu_gb300.workloads import water_box

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


# sizes whose groups are of 1, 2 and 8 molecules, and pools that mix them
POOLS = [[64, 333], [333, 2499, 64], [10001, 2499, 5], [7] * 400 + [333]]


@pytest.fixture(scope="module")
def alone(ctx):
    out = {}
    for n in sorted({n for p in POOLS for n in p}):
        bt = ChainBatch(ctx, [water_box(n, seed=n, cutoff=5.0 if n < 64 else 9.0,
                                        L=16.0 if n < 64 else None)], [1], rotation=ROT_AXIS)
        out[n] = bt.system_energies()[0]
        bt.close()
    return out


@pytest.mark.parametrize("pool", range(len(POOLS)))
def test_energy_does_not_depend_on_the_pool(ctx, alone, pool):
    sizes = POOLS[pool]
    boxes = [water_box(n, seed=n, cutoff=5.0 if n < 64 else 9.0, L=16.0 if n < 64 else None)
             for n in sizes]
    for order in (range(len(sizes)), range(len(sizes) - 1, -1, -1)):
        bt = ChainBatch(ctx, [boxes[i] for i in order], [1] * len(sizes), rotation=ROT_AXIS)
        e = bt.system_energies()
        for c, i in enumerate(order):
            assert e[c] == alone[sizes[i]], (c, sizes[i])
        bt.close()
