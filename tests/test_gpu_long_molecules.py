"""FP32 plain energies of one species around the length from which a neighbour's items
go entry by entry (16 atoms) and up to the longest, in boxes so small that many pairs
of molecules straddle half an edge: molecule energies, moves and the system energy
against the oracle by the FP32-pair rule (tol_mixed of the terms' magnitudes)."""
import numpy as np
import pytest

from helpers import tol_mixed
from mcgpu_gb300 import PREC_MIXED, Context, GpuBox
from oracle.pyoracle import OracleBox
from test_gpu_fp64_items import mixed_box, one_primary
from test_gpu_work_split import gentle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n_mol", [9, 41])
@pytest.mark.parametrize("length", [15, 16, 17, 31, 32, 33, 64])
def test_one_species(ctx, length, n_mol):
    box = gentle(one_primary(mixed_box(50 + length, n_mol, [length], (21.0, 17.0, 19.0), 8.4)))
    o, g = OracleBox(box), GpuBox(ctx, box, PREC_MIXED)
    r = o.system_energy()
    scale = sum(o.mol_energy_abs(m, m) for m in range(n_mol))
    assert abs(g.system_energy() - r) <= tol_mixed(r, scale)
    for m in range(n_mol):
        r = o.mol_energy(m, 0)
        assert abs(g.mol_energy(m, 0) - r) <= tol_mixed(r, o.mol_energy_abs(m, 0)), m
    rng = np.random.default_rng(length)
    for m in rng.integers(0, n_mol, 8):
        mv = (int(rng.integers(length)), *rng.uniform(-0.3, 0.3, 3), *rng.uniform(-20, 20, 3))
        r0, s0 = o.mol_energy(m, 0), o.mol_energy_abs(m, 0)
        o.apply_move(m, *mv)
        r1, s1 = o.mol_energy(m, 0), o.mol_energy_abs(m, 0)
        e0, e1 = g.move_energies(int(m), *mv)
        assert abs(e0 - r0) <= tol_mixed(r0, s0) and abs(e1 - r1) <= tol_mixed(r1, s1), m
    g.close()
