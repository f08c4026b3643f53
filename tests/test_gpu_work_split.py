"""The work splits of the FP32 pair paths, list builds and chain schedules where
they can go wrong, against the oracle: chains of one species whose ring entries
the warps share (1 to 64 atoms, a neighbour atom a lane; more hits than a warp's
ring holds at once); plain energies whose items are dealt over lanes (mixed
lengths, skipped sites, several primaries); list builds with cells of more
members than the sorted buffer, more candidates than one chunk, and too few
cells to skip any; volume moves of mixed lengths and of several primaries; more
chains than groups, in several segments.

Tolerances: decisions and coordinates equal; energies by the FP32-pair rule
(tol_mixed of the terms' magnitudes), volume energies as in the isobaric
replays."""
import numpy as np
import pytest

from helpers import tol_mixed
from mcgpu_gb300 import PREC_FP64, PREC_MIXED, ROT_AXIS, ChainBatch, Context, GpuBox
from mcgpu_gb300 import workloads as W
from oracle.pyoracle import OracleBox, OracleChain
from test_gpu_chain import check_energies, replay
from test_gpu_fp64_items import mixed_box, one_primary
from test_gpu_npt import oracle_npt, scale_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def gentle(box):
    """The molecules drawn together to half their size: no atoms of different
    molecules nearer than 2 A."""
    b = box.copy()
    first = np.repeat(b.mol_start, b.mol_len)
    for v in (b.x, b.y, b.z):
        a = v[first]
        L = float(b.size[0 if v is b.x else 1 if v is b.y else 2])
        d = v - a
        d -= L * np.round(d / L)
        v[:] = a + 0.5 * d
    return b.wrap()


def lattice(k: int, spacing: float, cutoff: float):
    """k^3 one-atom molecules on a cubic lattice."""
    L = k * spacing
    g = (np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5)
    t = (np.zeros((1, 3)), np.array([1.3]), np.array([0.1]), np.array([0.2]), 0)
    b = mixed_box(1, 1, [1], (L, L, L), cutoff)
    n = k ** 3
    b.x, b.y, b.z = (g * spacing).T.copy()
    b.sigma, b.epsilon, b.charge = (np.full(n, float(t[i][0])) for i in (1, 2, 3))
    b.mol_start, b.mol_len = np.arange(n), np.ones(n)
    b.mol_pidx_start, b.mol_pidx_count, b.pidx = np.arange(n), np.ones(n), np.arange(n)
    return b.normalise()


@pytest.mark.parametrize("tile", [(64, 2, 4), (128, 1, 16), (256, 2, 8)])
@pytest.mark.parametrize("length", [1, 2, 4, 5, 16, 64])
def test_one_species_chains(ctx, length, tile):
    box = gentle(one_primary(mixed_box(20 + length, 200, [length], (30.0, 30.0, 30.0), 14.9)))
    bt = ChainBatch(ctx, [box], [99], rotation=ROT_AXIS)
    bt.set_tile(*tile)
    tr = bt.run_traced(80)[0]
    oc, _, otr, _, _ = replay(box, 99, 0, tr, ROT_AXIS)
    check_energies(box, tr, otr, ROT_AXIS, 99, 0)
    assert np.array_equal(np.stack(bt.download(0), 1), oc.coords())
    bt.close()


@pytest.mark.parametrize("lens,edges,single", [
    ([1, 2, 3, 5, 9, 16, 33, 64], (22.0, 22.0, 22.0), False),
    ([3, 9], (20.0, 26.0, 31.0), True), ([7], (19.0, 19.0, 19.0), False),
    ([64], (23.0, 23.0, 23.0), True)])
def test_plain_energies_fp32_pairs(ctx, lens, edges, single):
    box = gentle(mixed_box(31, 40, lens, edges, 9.4))
    if single:
        box = one_primary(box)
    o, g = OracleBox(box), GpuBox(ctx, box, PREC_MIXED)
    rng = np.random.default_rng(3)
    for m in range(box.n_mol):
        r = o.mol_energy(m, 0)
        assert abs(g.mol_energy(m, 0) - r) <= tol_mixed(r, o.mol_energy_abs(m, 0)), m
    for m in rng.integers(0, box.n_mol, 8):
        mv = (int(rng.integers(box.mol_len[m])), *rng.uniform(-0.3, 0.3, 3),
              *rng.uniform(-20, 20, 3))
        r0, s0 = o.mol_energy(m, 0), o.mol_energy_abs(m, 0)
        o.apply_move(m, *mv)
        r1, s1 = o.mol_energy(m, 0), o.mol_energy_abs(m, 0)
        e0, e1 = g.move_energies(int(m), *mv)
        assert abs(e0 - r0) <= tol_mixed(r0, s0) and abs(e1 - r1) <= tol_mixed(r1, s1), m
    g.close()


@pytest.mark.parametrize("k,spacing,cutoff,skin", [
    (20, 1.5, 8.5, 1.0),    # 27 cells of 296 members, 8,000 candidates
    (12, 2.0, 10.5, 1.4),   # two cells an edge: every cell is a neighbour
    (9, 3.5, 5.0, 1.0)])    # five cells an edge
def test_list_builds(ctx, k, spacing, cutoff, skin):
    boxes = [lattice(k, spacing, cutoff), lattice(max(k - 4, 4), spacing, min(cutoff, 4.0))]
    bt = ChainBatch(ctx, boxes, [5, 6], rotation=ROT_AXIS)
    bt.set_tile(128, 1, 16)
    bt.set_verlet(skin)
    tr = bt.run_traced(60)
    for c, b in enumerate(boxes):
        oc, _, _, _, _ = replay(b, [5, 6][c], c, tr[c], ROT_AXIS)
        assert np.array_equal(np.stack(bt.download(c), 1), oc.coords())
        assert bt.stats()[c].nl_builds >= 1
    bt.close()


def test_volume_moves_of_mixed_lengths(ctx):
    """One and several primaries, uneven edges, cutoffs near half an edge."""
    boxes = [gentle(mixed_box(41, 60, [1, 2, 3, 5, 9, 16, 33, 64], (26.0, 26.0, 26.0), 9.0)),
             gentle(one_primary(mixed_box(42, 50, [3, 9], (22.0, 24.0, 27.0), 10.9))),
             gentle(one_primary(mixed_box(43, 90, [5], (40.0, 40.0, 40.0), 8.0))),
             gentle(mixed_box(44, 2, [7, 4], (20.0, 20.0, 20.0), 9.0))]
    seeds, interval, steps, dl = [1, 2, 3, 4], 10, 80, 0.02
    bt = ChainBatch(ctx, boxes, seeds, rotation=ROT_AXIS)
    bt.set_tile(128, 1, 16)
    bt.set_npt(interval, 1.0, dl, PREC_MIXED)
    tr, vtr = bt.run_traced(steps, volume=True)
    for c, b in enumerate(boxes):
        oc, _, otr, ovol = oracle_npt(b, seeds[c], c, steps, interval, 1.0, dl)
        for s, (t, r) in enumerate(zip(tr[c], otr)):
            assert t.mol == r.mol and bool(t.accepted) == bool(r.accepted), (c, s)
        for k, (t, r) in enumerate(zip(vtr[c], ovol)):
            assert bool(t.accepted) == (r["status"] == 1), (c, k)
            assert t.edge == r["edge"], (c, k)
            if t.evaluated:
                tight = 1e-11 * max(1.0, abs(r["e_old"]))
                loose = 2e-6 * max(abs(r["e_old"]), 1e-3 * scale_of(oc.ob, b))
                assert abs(t.e_new - r["e_new"]) <= (tight if t.fp64 else loose), (c, k)
        assert np.array_equal(np.stack(bt.download(c), 1), oc.coords()), c
    bt.close()


@pytest.mark.parametrize("tile", [(128, 1, 16), (256, 4, 8)])
def test_more_chains_than_groups(ctx, tile):
    """1,400 chains of 4 to 60 molecules in segments of 16 steps and a short last
    one: every chain takes every step once, and a sample of them is the oracle's."""
    rng = np.random.default_rng(9)
    sizes = rng.integers(4, 61, 1400)
    kinds = {int(n): W.water_box(int(n), seed=int(n)) for n in set(sizes.tolist())}
    for b in kinds.values():
        b.cutoff = min(b.cutoff, 0.5 * float(b.size[0]))
    boxes = [kinds[int(n)] for n in sizes]
    seeds = list(range(100, 100 + len(boxes)))
    bt = ChainBatch(ctx, boxes, seeds, rotation=ROT_AXIS)
    bt.set_tile(*tile)
    bt.run(16 * 3 + 5)
    bt.run(7)
    stats = bt.stats()
    assert all(s.steps == 60 and s.error == 0 for s in stats)
    for c in rng.integers(0, len(boxes), 12):
        oc = OracleChain(boxes[c], ROT_AXIS)
        _, acc, _ = oc.run(seeds[c], int(c), 60, oc.system_energy())
        assert stats[c].accepted == acc
        assert np.array_equal(np.stack(bt.download(int(c)), 1), oc.coords()), c
    bt.close()


@pytest.mark.parametrize("n,skin,interval", [(37, 0.0, 0), (60, 0.0, 0), (3, 1.0, 0),
                                             (20, 0.0, 15), (4, 1.0, 15)])
def test_few_fp64_chains_equal_many(ctx, n, skin, interval):
    """Few FP64-pair chains run in windows over clusters, many one step at a time:
    the same chains, decisions and coordinates (FP64 sums in another order), also
    from a checkpoint restored into a batch whose precision was not set."""
    boxes, seeds = W.water_chains(80, n_min=300 if skin else 40, n_max=400, seed=23)
    def batch(k, f64=True):
        bt = ChainBatch(ctx, boxes[:k], seeds[:k], rotation=ROT_AXIS)
        bt.set_tile(128, 1, 16)
        if f64:
            bt.set_precision(PREC_FP64)
        if interval:
            bt.set_npt(interval, 1.0, 0.02)
        if skin:
            bt.set_verlet(skin)
        return bt
    many, few = batch(80), batch(n)
    for bt in (many, few):
        bt.run(40)
    ck = few.checkpoint()
    again = batch(n, False)
    again.restore(ck)
    for bt in (many, few, again):
        bt.run(33)
    sm = many.stats()
    for bt in (few, again):
        for c, s in enumerate(bt.stats()):
            assert (s.accepted, s.steps, s.error) == (sm[c].accepted, 73, 0), c
            assert (s.ties, s.pairs) == (sm[c].ties, sm[c].pairs), c
            assert s.window_redo == 0 and s.vol_accepted == sm[c].vol_accepted
            assert abs(s.energy - sm[c].energy) <= 1e-9 * max(1.0, abs(sm[c].energy)), c
            assert np.array_equal(np.stack(bt.download(c)), np.stack(many.download(c))), c
    for bt in (many, few, again):
        bt.close()
