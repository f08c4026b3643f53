"""FP64 system energies of boxes large enough that a CTA sums several molecules
(from 2,432 on two, from 9,728 on eight) where those molecules are not alike: their
lengths differ, or one length has its skipped sites at different places.  A warp's
lanes then hold rows of different trip counts.  Every entry point that forms such a
sum, against the oracle.

FP64 pair terms in another order: tol64 (1e-11 of the sum of the terms'
magnitudes weighted by their condition numbers)."""
import numpy as np
import pytest

from helpers import tol64
from mcgpu_gb300 import (PREC_FP64, PREC_MIXED, ROT_AXIS, ChainBatch, Context, GpuBox,
                         run_plain_device_many)
from oracle.pyoracle import OracleBox, OracleChain
from test_gpu_fp64_items import device_energy, mixed_box, one_primary

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def two_patterns(box):
    """Molecules of 7 atoms: every other one skips its third site beside the last."""
    box = box.copy()
    box.sigma[box.mol_start[1::2] + 2] = -1.0
    return box.normalise()


BOXES = {
    "3_and_9": lambda: mixed_box(31, 2500, [3, 9], (84.0, 84.0, 84.0), 9.0),
    "1_to_64": lambda: mixed_box(32, 2433, [64, 1, 33, 2, 16, 3, 9, 5], (86.0, 83.0, 90.0), 8.0),
    "solute": lambda: mixed_box(33, 2432, [3] * 1215 + [40] + [3] * 1216, (84.0,) * 3, 9.0),
    "two_patterns": lambda: two_patterns(mixed_box(34, 2434, [7], (84.0,) * 3, 9.0)),
    "groups_of_8": lambda: mixed_box(35, 9731, [3, 9, 1, 5, 3], (132.0,) * 3, 9.0),
}


@pytest.mark.parametrize("name", sorted(BOXES))
def test_system_energies(ctx, name):
    box = BOXES[name]()
    o = OracleBox(box)
    ref = o.system_energy()
    tol = tol64(ref, sum(o.mol_energy_abs(m, m) for m in range(0, box.n_mol, 7)))
    assert abs(device_energy(box) - ref) <= tol
    g = GpuBox(ctx, box, PREC_FP64)
    e = g.system_energy()
    assert abs(e - ref) <= tol
    # the device loop's start
    assert run_plain_device_many([g], [5], 0)[0].energy0 == e
    # the host loop's start and its drift over a few moves
    st = g.run_plain_native(3, 8, True)
    assert abs(st.energy0 - ref) <= tol
    assert abs(st.energy - g.system_energy()) <= tol
    g.close()


@pytest.mark.parametrize("name", ["3_and_9", "solute"])
def test_chain_start(ctx, name):
    """A device-resident run starts from the FP64 system energy of its own coordinates
    (the box's in fixed point, as the oracle's chain holds them)."""
    box = one_primary(BOXES[name]())
    g = GpuBox(ctx, box, PREC_MIXED)
    st, tr = g.chain_run(seed=11, n_steps=4, trace=True)
    o = OracleBox(box)
    ref = OracleChain(box, ROT_AXIS).system_energy()
    tol = tol64(ref, sum(o.mol_energy_abs(m, m) for m in range(0, box.n_mol, 7)))
    moved = sum(t.de for t in tr if t.accepted)
    # the changes themselves are FP32 sums added in double-float
    assert abs(st.energy - ref - moved) <= tol + 1e-6 * max(1.0, abs(moved))
    g.close()


def test_batch_pool(ctx):
    """Chains of unlike molecules, few each, many in the pool."""
    boxes = [one_primary(mixed_box(40 + c, 300 + c, [3, 9, 1, 64], (42.0,) * 3, 9.0))
             for c in range(9)]
    bt = ChainBatch(ctx, boxes, list(range(9)), rotation=ROT_AXIS)
    e = bt.system_energies()
    for c, b in enumerate(boxes):
        b = b.copy()
        b.x, b.y, b.z = bt.download(c)
        o = OracleBox(b)
        scale = sum(o.mol_energy_abs(m, m) for m in range(b.n_mol))
        assert abs(e[c] - o.system_energy()) <= tol64(o.system_energy(), scale), c
    bt.close()
