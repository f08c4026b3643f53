"""The FP64 pair batches (batch_items64, pair_sum64) and the grouped system
energies (k_pair_sums64, k_static_pair_sums) where their item
mapping and image choice can go wrong: molecules of 1 to 64 atoms in one
box (items found in prefix sums), one species (items by atom), partial and
full batches, several primaries, skipped sites, sites without LJ or charge,
edges that the cutoff nearly halves and boxes of unequal edges -- molecule
and system energies and moves of the plain path, and FP64-pair chains,
against the oracle.

FP64 pair terms in another order: tol64 (1e-11 of the sum of the terms'
magnitudes weighted by their condition numbers)."""
import numpy as np
import pytest

from helpers import tol64
from mcgpu_gb300 import PREC_FP64, ROT_AXIS, ChainBatch, Context, GpuBox
from mcgpu_gb300.workloads import BoxData, random_rotations, rsa_centres
from oracle.pyoracle import OracleBox, OracleChain

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def mixed_box(seed: int, n_mol: int, lens, edges, cutoff: float) -> BoxData:
    """n_mol rigid molecules of lens[m % len(lens)] atoms within 1.9 A of
    their centre, centres at least 4 A apart (atom pairs at least 0.2 A);
    every third site without LJ, every fifth without charge, every seventh
    skipped (negative sigma) except a molecule's first; one to three
    primaries."""
    rng = np.random.default_rng(seed)
    L = np.asarray(edges, float)
    centres = rsa_centres(seed, n_mol, float(L.min()), 4.0) * (L / L.min())
    rows = {k: [] for k in ("xyz", "sig", "eps", "q", "ms", "ml", "ps", "pc", "pidx")}
    at = 0
    for m in range(n_mol):
        n = lens[m % len(lens)]
        t = rng.normal(size=(n, 3))
        t *= (1.9 * rng.random((n, 1)) ** (1 / 3)) / np.linalg.norm(t, axis=1, keepdims=True)
        t = (t - t[0]) * 0.5          # first atom at the centre, others within 1.9 A
        k = np.arange(n)
        sig, eps = rng.uniform(0.5, 1.5, n), rng.uniform(0.01, 0.2, n)
        eps[k % 3 == 1] = 0.0
        sig[k % 6 == 4] = 0.0
        q = rng.uniform(-0.4, 0.4, n)
        q[k % 5 == 3] = 0.0
        sig[(k % 7 == 6)] = -1.0
        rows["xyz"].append(t @ random_rotations(rng, 1)[0].T + centres[m])
        rows["sig"].append(sig)
        rows["eps"].append(eps)
        rows["q"].append(q)
        np_ = min(n, 1 + m % 3)
        rows["ms"].append(at)
        rows["ml"].append(n)
        rows["ps"].append(len(rows["pidx"]))
        rows["pc"].append(np_)
        rows["pidx"].extend(range(at, at + np_))
        at += n
    xyz = np.concatenate(rows["xyz"])
    return BoxData(x=xyz[:, 0].copy(), y=xyz[:, 1].copy(), z=xyz[:, 2].copy(),
                   sigma=np.concatenate(rows["sig"]), epsilon=np.concatenate(rows["eps"]),
                   charge=np.concatenate(rows["q"]), mol_start=np.array(rows["ms"]),
                   mol_len=np.array(rows["ml"]), mol_pidx_start=np.array(rows["ps"]),
                   mol_pidx_count=np.array(rows["pc"]), pidx=np.array(rows["pidx"]),
                   size=L, cutoff=cutoff, temperature=300.0, max_translate=0.2,
                   max_rotate=15.0).normalise().wrap()


CASES = {
    "lengths_1_to_64": (1, 37, [1, 2, 3, 5, 9, 16, 33, 64], (22.0, 22.0, 22.0), 9.0),
    "uneven_edges": (2, 70, [3, 9], (20.0, 26.0, 31.0), 9.9),
    "one_atom": (3, 40, [1], (17.0, 17.0, 17.0), 8.4),
    "two_molecules": (4, 2, [7, 4], (18.0, 18.0, 18.0), 9.0),
    "one_species_5": (5, 67, [5], (24.0, 24.0, 24.0), 11.0),
}


def one_primary(box: BoxData) -> BoxData:
    """The same box with each molecule's first primary alone (a chain of one
    species then takes the items by atom)."""
    b = box.copy()
    b.pidx = b.pidx[b.mol_pidx_start].copy()
    b.mol_pidx_start = np.arange(b.n_mol)
    b.mol_pidx_count = np.ones(b.n_mol)
    sl = int(b.mol_len[0])
    if np.all(b.mol_len == sl):
        for k in ("sigma", "epsilon", "charge"):
            setattr(b, k, np.tile(getattr(b, k)[:sl], b.n_mol))
    return b.normalise()


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_energies_and_moves(ctx, name, single):
    box = mixed_box(*CASES[name])
    if single:
        box = one_primary(box)
    o, g = OracleBox(box), GpuBox(ctx, box, PREC_FP64)
    ref = o.system_energy()
    scale = sum(o.mol_energy_abs(m, m) for m in range(box.n_mol))
    assert abs(g.system_energy() - ref) <= tol64(ref, scale)
    rng = np.random.default_rng(7)
    for m in range(box.n_mol):
        r = o.mol_energy(m, 0)
        assert abs(g.mol_energy(m, 0) - r) <= tol64(r, o.mol_energy_abs(m, 0)), m
    for m in rng.integers(0, box.n_mol, 12):
        mv = (int(rng.integers(box.mol_len[m])), *rng.uniform(-0.5, 0.5, 3),
              *rng.uniform(-30, 30, 3))
        r0, s0 = o.mol_energy(m, 0), o.mol_energy_abs(m, 0)
        o.apply_move(m, *mv)
        r1, s1 = o.mol_energy(m, 0), o.mol_energy_abs(m, 0)
        e0, e1 = g.move_energies(int(m), *mv)
        assert abs(e0 - r0) <= tol64(r0, s0) and abs(e1 - r1) <= tol64(r1, s1), m
    assert np.array_equal(np.stack(g.download(), 1), o.coords())
    g.close()


@pytest.mark.parametrize("name", ["lengths_1_to_64", "one_species_5", "two_molecules"])
def test_fp64_chains(ctx, name):
    """FP64-pair chains: the oracle's decisions and coordinates."""
    box = one_primary(mixed_box(*CASES[name]))
    bt = ChainBatch(ctx, [box], [99], rotation=ROT_AXIS)
    bt.set_tile(128, 1, 16)
    from mcgpu_gb300 import PREC_FP64 as F64
    bt.set_precision(F64)
    tr = bt.run_traced(120)[0]
    oc = OracleChain(box, ROT_AXIS)
    _, _, otr = oc.run(99, 0, 120, oc.system_energy())
    for t, r in zip(tr, otr):
        assert t.mol == r.mol and bool(t.accepted) == bool(r.accepted)
        assert abs(t.de - r.de) <= 1e-9 * max(1.0, abs(r.e_old) + abs(r.e_new))
    assert np.array_equal(np.stack(bt.download(0), 1), oc.coords())
    bt.close()


def device_energy(box: BoxData) -> float:
    """mcgpu_system_energy_static over the box's rows in device memory."""
    import ctypes as C
    import torch
    from mcgpu_gb300 import _abi
    d, keep = _abi.BoxDesc(), []
    d.n_mol, d.n_atom, d.n_pidx = box.n_mol, box.n_atom, box.n_pidx
    for k in ("x", "y", "z", "sigma", "epsilon", "charge", "mol_start", "mol_len",
              "mol_pidx_start", "mol_pidx_count", "pidx"):
        t = torch.from_numpy(getattr(box, k).copy()).cuda()
        keep.append(t)
        kind = _abi._dp if t.dtype == torch.float64 else _abi._ip
        setattr(d, k, C.cast(C.c_void_p(t.data_ptr()), kind))
    for k in range(3):
        d.size[k] = float(box.size[k])
    d.cutoff = float(box.cutoff)
    out = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    _abi.check(_abi.lib().mcgpu_system_energy_static(
        C.byref(d), C.c_void_p(out.data_ptr()),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return float(out.item())


def unwrapped(box: BoxData) -> BoxData:
    """The box with whole molecules moved by up to three edges (the reference
    then takes its single shift of the raw difference)."""
    b = box.copy()
    rng = np.random.default_rng(11)
    for k, v in enumerate((b.x, b.y, b.z)):
        v += np.repeat(rng.integers(-3, 4, b.n_mol) * b.size[k], b.mol_len)
    return b


STATIC = {
    # molecules of more atoms than one stage holds, alone and beside short ones
    "long_molecules": lambda: mixed_box(6, 11, [70, 130, 3, 64], (22.0, 22.0, 22.0), 10.0),
    "unwrapped": lambda: unwrapped(mixed_box(7, 60, [3, 9, 1], (24.0, 24.0, 24.0), 9.0)),
    "one_molecule": lambda: mixed_box(8, 1, [4], (20.0, 20.0, 20.0), 9.0),
    "nine_molecules": lambda: mixed_box(9, 9, [5, 2], (20.0, 20.0, 20.0), 9.9),
}


@pytest.mark.parametrize("name", sorted(STATIC))
def test_static_rows(ctx, name):
    box = STATIC[name]()
    o = OracleBox(box)
    ref = o.system_energy()
    scale = sum(o.mol_energy_abs(m, m) for m in range(box.n_mol))
    assert abs(device_energy(box) - ref) <= tol64(ref, scale)


@pytest.mark.parametrize("n_mol", [2433, 2500, 9729])
def test_groups_of_molecules(ctx, n_mol):
    """Sizes at which a CTA takes 2 and 8 molecules (the last group short)."""
    from mcgpu_gb300.workloads import water_box
    box = water_box(n_mol, seed=n_mol)
    o = OracleBox(box)
    ref = o.system_energy()
    scale = sum(o.mol_energy_abs(m, m) for m in range(0, n_mol, 37)) * 37
    g = GpuBox(ctx, box, PREC_FP64)
    assert abs(g.system_energy() - ref) <= tol64(ref, scale)
    assert abs(device_energy(box) - ref) <= tol64(ref, scale)
    g.close()


def test_groups_that_span_chains(ctx):
    """A batch of many small chains: groups of molecules from several."""
    from mcgpu_gb300.workloads import WATER_DENSITY, water_box
    boxes = []
    for c in range(600):
        n = 8 + c % 7
        L = (n / WATER_DENSITY) ** (1 / 3)
        boxes.append(water_box(n, L=L, cutoff=L / 2, seed=c, dmin=2.0))
    bt = ChainBatch(ctx, boxes, list(range(600)), rotation=ROT_AXIS)
    e = bt.system_energies()
    for c in range(0, 600, 7):
        b = boxes[c].copy()
        b.x, b.y, b.z = bt.download(c)
        o = OracleBox(b)
        scale = sum(o.mol_energy_abs(m, m) for m in range(b.n_mol))
        assert abs(e[c] - o.system_energy()) <= tol64(o.system_energy(), scale), c
    bt.close()


@pytest.mark.parametrize("prec", [PREC_FP64, 1])
def test_many_boxes_start_energies(ctx, prec):
    """The device loop's start energies of boxes of uneven sizes, all in one
    launch: each the box's own system energy."""
    from mcgpu_gb300 import run_plain_device_many
    boxes = [GpuBox(ctx, one_primary(mixed_box(20 + i, 2 + 9 * i, [3, 5], (21.0, 21.0, 21.0), 9.0)),
                    prec) for i in range(5)]
    own = [b.system_energy() for b in boxes]
    st = run_plain_device_many(boxes, range(5), 0)
    for e, s in zip(own, st):
        assert s.energy0 == e and s.energy == e
    for b in boxes:
        b.close()
