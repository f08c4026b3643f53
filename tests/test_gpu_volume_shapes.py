"""Volume moves with FP32 pairs at sizes whose kernel runs one to eight warps a CTA, of
one species and of mixed lengths: a chain's energies and edges are the same, bit for
bit, alone and in a batch with chains of the other kind (the kernel is then the one for
mixed lengths), and the mixed chains' energies the oracle's by the FP32-pair rule."""
import numpy as np
import pytest

from helpers import tol_mixed
from mcgpu_gb300 import PREC_MIXED, ROT_AXIS, ChainBatch, Context
from mcgpu_gb300.workloads import water_box
from oracle.pyoracle import OracleBox
from test_gpu_fp64_items import mixed_box, one_primary
from test_gpu_work_split import gentle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def run(ctx, boxes):
    """Every chain has its own key; chain ids follow the place, so equal places only."""
    bt = ChainBatch(ctx, boxes, [9 + c for c in range(len(boxes))], rotation=ROT_AXIS)
    bt.set_tile(64, 1, 20)
    bt.set_npt(20, 1.0, 0.004, PREC_MIXED)
    bt.run(100)
    out = [(s.energy, tuple(s.box), s.vol_accepted, s.accepted) for s in bt.stats()]
    xyz = [np.stack(bt.download(c), 1) for c in range(len(boxes))]
    bt.close()
    return out, xyz


@pytest.mark.parametrize("n", [20, 300, 700, 1500])
def test_one_species_beside_mixed_lengths(ctx, n):
    water = water_box(n, cutoff=6.0, seed=n)
    mixed = gentle(one_primary(mixed_box(60, 40, [3, 64, 9, 1], (26.0, 26.0, 26.0), 8.0)))
    alone, _ = run(ctx, [water])
    both, xyz = run(ctx, [water, mixed])
    assert both[0] == alone[0]
    b = mixed.copy()
    b.x, b.y, b.z = (np.ascontiguousarray(v) for v in xyz[1].T)
    b.size = np.array(both[1][1])
    o = OracleBox(b.normalise())
    scale = sum(o.mol_energy_abs(m, m) for m in range(b.n_mol))
    assert abs(both[1][0] - o.system_energy()) <= tol_mixed(o.system_energy(), scale)
    assert both[1][2] > 0
