"""The work that a user of this framework has it do, as measurable cases.

Every case goes through the public entry points: the SimulationStep contract
(``GpuBox.mol_energy``, ``system_energy`` and the host loop over them), the
reference's loop on the device, the device-resident chains (one large chain,
batches, NPT), the job server, and the system energy over rows the caller
holds.  Sizes, cutoffs, moves and temperatures are those of the repository's
own workloads: TIP3P-like water of 64 to 32,768 molecules, the rigid 16-atom
bicyclic molecule, and the flexible amine / water mixture.

Energies summed from FP64 pair terms are returned in FP64.  Those of the
mixed forms are sums of FP32 pair terms, so they are returned in FP32, the
precision they carry; coordinates, counts and decisions are exact either way.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import mcgpu_gb300 as M
from mcgpu_gb300 import _abi
from mcgpu_gb300.prepare import relax, tile_box

KT_PER_KELVIN = 0.00198717      # kcal/mol/K, the reference's constant
COULOMB = 332.06                # kcal A / mol / e^2, the reference's constant
FLOPS_PER_PAIR = 38             # distance 20, LJ with blending 12, Coulomb 4, sums 2
ATOMS = {"water": 3, "bicyclic": 16}
DENSITY = {"water": M.workloads.WATER_DENSITY, "bicyclic": M.workloads.BICYCLIC_DENSITY}
MOVES = {"water": (0.15, 15.0), "bicyclic": (0.2, 10.0)}


def listed() -> list[dict]:
    return [
        # The smallest call of the contract: one molecule's energy with its
        # neighbours, as a caller's own loop asks for it (latency).
        dict(name="molecule_water256_fp64", kind="molecule", species="water", n_mol=256,
             cutoff=9.0, precision="fp64"),
        # The drop-in: the reference's loop over the contract calls, its own
        # precision, on the 256-water box.
        dict(name="host_loop_water256_fp64", kind="host_loop", species="water", n_mol=256,
             cutoff=9.0, precision="fp64", steps=200, fused=False),
        # The drop-in on the single-chain workload (4000 16-atom molecules)
        # with FP32 pairs and one launch a move.
        dict(name="host_loop_bicyclic4000_mixed", kind="host_loop", species="bicyclic",
             n_mol=4000, cutoff=12.0, precision="mixed", steps=200, fused=True),
        # The reference's loop on the device with its rand() stream, one box.
        dict(name="device_loop_water256_fp64", kind="device_loop", species="water", n_mol=256,
             cutoff=9.0, precision="fp64", steps=400, boxes=1),
        # An ensemble of flexible molecules: bonds and angles move too.
        dict(name="device_loop_flex512x304_fp64", kind="device_loop", species="flex",
             n_mol=512, cutoff=0.0, precision="fp64", steps=192, boxes=304),
        # One large chain of many-atom molecules over several SMs.
        dict(name="chain_bicyclic4000_window16", kind="chain", species="bicyclic", n_mol=4000,
             cutoff=12.0, steps=1024, warm=64, skin=1.5, window=16),
        # The headline: 512 independent water chains of uneven size.
        dict(name="batch_water512", kind="batch", species="water", chains=512, n_min=64,
             n_max=2048, steps=1280, warm=1600, precision="mixed"),
        # A few chains of odd sizes with FP64 pairs on every step.
        dict(name="batch_water37_fp64", kind="batch", species="water", chains=37, n_min=64,
             n_max=700, steps=96, warm=32, precision="fp64"),
        # The large system at constant pressure: Verlet lists, windows of 8
        # steps, a volume move every 500 steps.
        dict(name="npt_water32768_window8", kind="npt", tiles=4, cutoff=12.0, steps=1000,
             warm=100, interval=500, skin=1.5, window=8),
        # A server's load: isobaric jobs of both species, many sizes.
        dict(name="served_jobs160", kind="served", jobs=160, n_min=128, n_max=4096, steps=2500),
        # The total energy of the large system (start, drift checks), FP64.
        dict(name="system_energy_water32768_fp64", kind="system", species="water", n_mol=32768,
             cutoff=12.0, precision="fp64"),
        # The total energy over rows in the caller's own device memory, an odd
        # number of 16-atom molecules.
        dict(name="static_energy_bicyclic1999", kind="static", species="bicyclic", n_mol=1999,
             cutoff=12.0),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["molecule", "host_loop", "device_loop", "flex", "chain", "batch", "batch64",
                       "npt", "served", "system", "static"])
    species = rng.choice(["water", "water", "bicyclic"])
    rc = 9.0 if species == "water" else 12.0
    top = {"water": 32768, "bicyclic": 4000}[species]
    if kind == "molecule":
        return dict(kind="molecule", species=species, n_mol=_log_int(rng, 128, top), cutoff=rc,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "host_loop":
        return dict(kind="host_loop", species=species, n_mol=_log_int(rng, 128, 4000), cutoff=rc,
                    precision=rng.choice(["fp64", "mixed"]), steps=rng.randrange(40, 200),
                    fused=rng.random() < 0.5)
    if kind == "device_loop":
        return dict(kind="device_loop", species=species, n_mol=_log_int(rng, 128, 1024), cutoff=rc,
                    precision=rng.choice(["fp64", "mixed"]), steps=rng.randrange(60, 200),
                    boxes=_log_int(rng, 1, 32))
    if kind == "flex":
        return dict(kind="device_loop", species="flex", n_mol=2 * _log_int(rng, 24, 256),
                    cutoff=0.0, precision=rng.choice(["fp64", "mixed"]),
                    steps=rng.randrange(40, 128), boxes=_log_int(rng, 1, 152))
    if kind == "chain":
        return dict(kind="chain", species=species, n_mol=_log_int(rng, 512, min(top, 8192)),
                    cutoff=rc, steps=rng.randrange(300, 1024), warm=64,
                    skin=rng.choice([0.0, 1.0, 1.5]), window=rng.choice([1, 4, 8, 16]))
    if kind in ("batch", "batch64"):
        f64 = kind == "batch64"
        return dict(kind="batch", species=species, chains=_log_int(rng, 3, 48 if f64 else 512),
                    n_min=64 if species == "water" else 128,
                    n_max=_log_int(rng, 256, 700 if f64 else 2048 if species == "water" else 1024),
                    steps=rng.randrange(48, 96) if f64 else rng.randrange(200, 1000),
                    warm=32 if f64 else 500, precision="fp64" if f64 else "mixed")
    if kind == "npt":
        return dict(kind="npt", tiles=rng.choice([2, 3, 4]), cutoff=rng.choice([9.0, 10.5, 12.0]),
                    steps=rng.randrange(500, 1000), warm=100, interval=rng.choice([250, 400, 500]),
                    skin=rng.choice([1.0, 1.5, 2.0]), window=rng.choice([1, 4, 8]))
    if kind == "served":
        return dict(kind="served", jobs=_log_int(rng, 8, 160), n_min=128,
                    n_max=_log_int(rng, 1024, 4096), steps=rng.randrange(300, 2500))
    if kind == "system":
        return dict(kind="system", species=species, n_mol=_log_int(rng, 256, top), cutoff=rc,
                    precision=rng.choice(["fp64", "mixed"]))
    return dict(kind="static", species=species, n_mol=_log_int(rng, 256, min(top, 8192)),
                cutoff=rc)


# ---- inputs -----------------------------------------------------------------------

def _box(ctx, species: str, n_mol: int, cutoff: float, seed: int) -> M.BoxData:
    """A box of the named species at its density, 298 K.  Water from random
    centres; boxes of up to 2048 relaxed by some sweeps of the chain, so that
    their energies are a liquid's.  The bicyclic molecule on its FCC lattice."""
    if species == "bicyclic":
        box = M.bicyclic_box(n_mol, cutoff=cutoff, seed=seed, lattice=True)
    else:
        box = M.water_box(n_mol, cutoff=cutoff, temperature=298.0, seed=seed)
    box.cutoff = min(box.cutoff, 0.5 * float(box.size[0]))
    if ctx is not None and species == "water" and n_mol <= 2048:
        box = relax(ctx, box, seed, 20 * n_mol)
    return box


def _flex_box(n_mol: int, seed: int):
    """The flexible mixture with every molecule shifted a little."""
    box, topo = M.workloads.flex_amine_water(n_mol)
    rng = np.random.default_rng(seed)
    shift = np.repeat(rng.uniform(-0.05, 0.05, (box.n_mol, 3)), box.mol_len, axis=0)
    box.x, box.y, box.z = box.x + shift[:, 0], box.y + shift[:, 1], box.z + shift[:, 2]
    return box.normalise().wrap(), topo


def _precision(case) -> int:
    return M.PREC_FP64 if case["precision"] == "fp64" else M.PREC_MIXED


class _DeviceRows:
    """A box's rows in device memory that the caller owns."""

    def __init__(self, box: M.BoxData):
        self.rows = {}
        d = _abi.BoxDesc()
        d.n_mol, d.n_atom, d.n_pidx = box.n_mol, box.n_atom, box.n_pidx
        for k in ("x", "y", "z", "sigma", "epsilon", "charge", "mol_start", "mol_len",
                  "mol_pidx_start", "mol_pidx_count", "pidx"):
            t = torch.from_numpy(getattr(box, k).copy()).cuda()
            self.rows[k] = t
            kind = _abi._dp if t.dtype == torch.float64 else _abi._ip
            setattr(d, k, ctypes.cast(ctypes.c_void_p(t.data_ptr()), kind))
        for k in range(3):
            d.size[k] = float(box.size[k])
        d.cutoff = float(box.cutoff)
        self.desc = d
        self.out = torch.zeros(1, dtype=torch.float64, device="cuda")


def _sizes(case, count: int, order: int) -> np.ndarray:
    """`count` sizes spread evenly over the logarithm of [n_min, n_max], in a
    mixed order (the same for every seed)."""
    n = np.exp(np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), count))
    return np.random.default_rng(order).permutation(np.rint(n).astype(int))


def _batch_boxes(case, seed: int):
    """Independent chains of one species at its density, 280 to 360 K."""
    rng = np.random.default_rng(seed)
    sizes = _sizes(case, case["chains"], 1)
    if case["species"] == "water":
        boxes = [_box(None, "water", int(n), 9.0, seed * 100003 + c) for c, n in enumerate(sizes)]
    else:
        few = [_box(None, "bicyclic", int(n), 12.0, seed + i)
               for i, n in enumerate(_sizes(case, 4, 1))]
        boxes = [few[c % 4].copy() for c in range(case["chains"])]
    for b in boxes:
        b.temperature = float(rng.uniform(280.0, 360.0))
    return boxes, rng.integers(1, 2 ** 63 - 1, case["chains"]).astype(np.uint64)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = {"case": case, "seed": int(seed)}
    if kind == "static":
        s["rows"] = _DeviceRows(_box(None, case["species"], case["n_mol"], case["cutoff"], seed))
        return s
    ctx = s["ctx"] = M.Context(0)
    if kind in ("molecule", "host_loop", "system"):
        box = _box(ctx, case["species"], case["n_mol"], case["cutoff"], seed)
        s["box"] = M.GpuBox(ctx, box, _precision(case))
        s["mol"] = int(seed) % case["n_mol"]
    elif kind == "device_loop" and case["species"] == "flex":
        s["boxes"] = []
        for i in range(case["boxes"]):
            if i % 8 == 0:
                box, topo = _flex_box(case["n_mol"], seed * 1009 + i)
            g = M.GpuBox(ctx, box, _precision(case))
            g.set_topology(topo)
            g.set_intra(True)
            s["boxes"].append(g)
    elif kind == "device_loop":
        boxes = [_box(ctx, case["species"], case["n_mol"], case["cutoff"], seed * 17 + i)
                 for i in range(min(case["boxes"], 4))]
        s["boxes"] = [M.GpuBox(ctx, boxes[i % len(boxes)], _precision(case))
                      for i in range(case["boxes"])]
    elif kind == "chain":
        box = _box(None, case["species"], case["n_mol"], case["cutoff"], seed)
        g = s["box"] = M.GpuBox(ctx, box, M.PREC_MIXED)
        if case["skin"] > 0:
            g.set_verlet(case["skin"])
        g.set_window(case["window"])
        g.chain_run(seed=seed, n_steps=case["warm"])
    elif kind == "batch":
        boxes, seeds = _batch_boxes(case, seed)
        bt = s["batch"] = M.ChainBatch(ctx, boxes, seeds, rotation=M.ROT_AXIS)
        bt.set_precision(_precision(case))
        bt.autotune(64 if case["precision"] == "mixed" else 16)
        bt.run(case["warm"])
    elif kind == "npt":
        small = M.water_box(512, L=99.3 / 4, cutoff=9.0, temperature=298.0, seed=seed)
        box = tile_box(relax(ctx, small, seed, 20 * 512), case["tiles"])
        box.cutoff = case["cutoff"]
        bt = s["batch"] = M.ChainBatch(ctx, [box], [seed * 7919 + 1], rotation=M.ROT_AXIS)
        bt.set_tile(512, 1, 64)
        bt.set_window(case["window"])
        bt.set_verlet(case["skin"])
        bt.set_npt(case["interval"], 1.0, 0.0015, M.PREC_MIXED)
        bt.run(case["warm"])
    elif kind == "served":
        rng = np.random.default_rng(seed)
        pool = [_box(None, species, int(n), rc, seed + k)
                for species, rc, order in (("water", 9.0, 2), ("bicyclic", 12.0, 3))
                for k, n in enumerate(_sizes(case, 6, order))]
        s["jobs"] = []
        for i in range(case["jobs"]):
            b = pool[(5 * i) % len(pool)].copy()
            b.temperature = float(rng.uniform(280.0, 360.0))
            s["jobs"].append((b, int(rng.integers(1, 2 ** 63))))
        s["server"] = M.JobServer(ctx, hbm_budget_bytes=8 << 30, max_slots=256, round_steps=100,
                                  max_mol_atoms=16, max_atoms=8_000_000, max_molecules=1_000_000)
    return s


# ---- one pass -----------------------------------------------------------------------

def _energy(case, e):
    """An energy at the precision of its pair terms."""
    e = np.asarray(e, np.float64)
    return e if case.get("precision") == "fp64" else e.astype(np.float32)


def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "molecule":
        return {"energy": _energy(case, s["box"].mol_energy(s["mol"], 0))}
    if kind == "host_loop":
        st = s["box"].run_plain_native(s["seed"] & 0xFFFF, case["steps"], case["fused"])
        return {"energy": _energy(case, st.energy), "accepted": int(st.accepted),
                "xyz": np.stack(s["box"].download(), 1)}
    if kind == "device_loop":
        st = M.run_plain_device_many(s["boxes"], [s["seed"] % 65521 + i
                                                  for i in range(len(s["boxes"]))], case["steps"])
        return {"energy": _energy(case, [v.energy for v in st]),
                "accepted": np.array([v.accepted for v in st]),
                "xyz": np.concatenate([np.stack(g.download(), 1) for g in s["boxes"]])}
    if kind == "chain":
        st, _ = s["box"].chain_run(seed=s["seed"], n_steps=case["steps"])
        return {"energy": _energy(case, st.energy), "accepted": int(st.accepted),
                "xyz": np.stack(s["box"].download(), 1)}
    if kind in ("batch", "npt"):
        bt = s["batch"]
        bt.run(case["steps"])
        st = bt.stats()
        xyz = bt.download_all()
        # the running energies of a batch start from FP32 pair sums whatever
        # its steps take; the chains' coordinates are views of three arrays
        # of the whole batch
        out = {"energy": np.array([v.energy for v in st], np.float32),
               "accepted": np.array([v.accepted for v in st]),
               "xyz": [v.base for v in xyz[0]]}
        if kind == "npt":
            out["edges"] = np.array([list(v.box) for v in st])
            out["volume_accepted"] = np.array([v.vol_accepted for v in st])
        return out
    if kind == "served":
        srv = s["server"]
        ids = [srv.submit(b, key, case["steps"], chain_id=i, npt=True, pressure_atm=1.0,
                          max_dlnv=0.01, vol_precision=M.PREC_MIXED)
               for i, (b, key) in enumerate(s["jobs"])]
        srv.drain()
        done = srv.results()
        res = [done[i].result for i in ids]
        return {"energy": _energy(case, [r.energy for r in res]),
                "accepted": np.array([r.accepted for r in res]),
                "edges": np.array([list(r.box) for r in res]),
                "xyz": np.concatenate([done[i].coords for i in ids])}
    if kind == "system":
        return {"energy": _energy(case, s["box"].system_energy())}
    rows = s["rows"]
    _abi.check(_abi.lib().mcgpu_system_energy_static(
        ctypes.byref(rows.desc), ctypes.c_void_p(rows.out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"energy": rows.out}


# ---- what a pass cannot do without ----------------------------------------------------

def _neighbours(density: float, n_mol: int, cutoff: float) -> float:
    L = (n_mol / density) ** (1 / 3)
    return min(n_mol - 1.0, density * 4.18879 * min(cutoff, 0.5 * L) ** 3)


def work(case: dict) -> dict:
    kind = case["kind"]
    flops = bytes_ = 0.0
    if case.get("species") == "flex":
        # half the molecules of 9 atoms, half of 3; pairs at both placements
        rho = 48 / 19.0 ** 3
        pairs = _neighbours(rho, case["n_mol"], 9.0) * 6 * 6
        moves = case["steps"] * case["boxes"]
        atoms = 6 * case["n_mol"] * case["boxes"]
        return {"flops": moves * 2 * (pairs + 36) * FLOPS_PER_PAIR, "bytes": atoms * (72 + 24)}
    if kind in ("molecule", "system", "static", "host_loop", "device_loop", "chain", "npt"):
        species = case.get("species", "water")
        n = case["n_mol"] if "n_mol" in case else 512 * case["tiles"] ** 3
        a = ATOMS[species]
        pairs = _neighbours(DENSITY[species], n, case["cutoff"]) * a * a
        boxes = case.get("boxes", 1)
        total = 0.5 * n * pairs * FLOPS_PER_PAIR
        bytes_ = boxes * n * a * 6 * 8.0 + 8
        if kind == "molecule":
            flops = pairs * FLOPS_PER_PAIR
        elif kind in ("system", "static"):
            flops = total
        else:
            flops = boxes * case["steps"] * 2 * pairs * FLOPS_PER_PAIR
            bytes_ += boxes * n * a * 3 * 8.0
            if kind in ("host_loop", "device_loop"):
                flops += boxes * total
            if kind == "npt":
                flops += 2 * total * (case["steps"] // case["interval"])
    else:
        many = case["chains"] if kind == "batch" else case["jobs"]
        mean_n = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        kinds = [case["species"]] if kind == "batch" else ["water", "bicyclic"]
        for species in kinds:
            a, k = ATOMS[species], many / len(kinds)
            rc = 9.0 if species == "water" else 12.0
            pairs = _neighbours(DENSITY[species], mean_n, rc) * a * a
            flops += k * case["steps"] * 2 * pairs * FLOPS_PER_PAIR
            bytes_ += k * mean_n * a * 9 * 8.0
            if kind == "served":
                flops += k * (case["steps"] // 100) * mean_n * pairs * FLOPS_PER_PAIR
    return {"flops": flops, "bytes": bytes_}


# ---- the same in plain 64-bit arithmetic ------------------------------------------------

class _Exact:
    """A box of one rigid species (one primary atom per molecule) in FP64."""

    def __init__(self, box: M.BoxData):
        self.n, self.a = box.n_mol, int(box.mol_len[0])
        self.pos = np.stack([box.x, box.y, box.z], 1).reshape(self.n, self.a, 3).copy()
        self.prim = int(box.pidx[0])
        self.L, self.rc2 = np.array(box.size), float(box.cutoff) ** 2
        self.kT = box.temperature * KT_PER_KELVIN
        self.max_t, self.max_r = box.max_translate, box.max_rotate
        sig, eps, q = (v[:self.a] for v in (box.sigma, box.epsilon, box.charge))
        self.sig2 = np.outer(sig, sig)
        self.eps4 = 4.0 * np.sqrt(np.outer(eps, eps))
        self.qq = np.outer(q, q) * COULOMB

    def image(self, d):
        return d - self.L * ((d > 0.5 * self.L).astype(float) - (d < -0.5 * self.L))

    def molecule(self, m: int, x: np.ndarray) -> float:
        """Energy of molecule m at coordinates x with every other molecule."""
        d = self.image(self.pos[:, self.prim] - x[self.prim])
        near = np.einsum("ij,ij->i", d, d) <= self.rc2
        near[m] = False
        d = self.image(self.pos[near][:, :, None, :] - x[None, None])
        r2 = np.einsum("ijkl,ijkl->ijk", d, d)
        s6 = (self.sig2 / r2) ** 3
        return float(np.sum(self.eps4 * (s6 * s6 - s6) + self.qq / np.sqrt(r2)))

    def system(self) -> float:
        """Energy of every pair of molecules once."""
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)
        pos, L, sig2, eps4, qq = map(t, (self.pos, self.L, self.sig2, self.eps4, self.qq))
        image = lambda d: d - L * ((d > 0.5 * L).double() - (d < -0.5 * L).double())
        prim, order, total = pos[:, self.prim], torch.arange(self.n, device=dev), 0.0
        for i0 in range(0, self.n, 256):
            i = order[i0:i0 + 256]
            d = image(prim[None] - prim[i][:, None])
            near = ((d * d).sum(-1) <= self.rc2) & (order[None] > i[:, None])
            ii, jj = near.nonzero(as_tuple=True)
            for k in range(0, ii.numel(), 1 << 16):
                d = image(pos[jj[k:k + (1 << 16)]][:, :, None] -
                          pos[i[ii[k:k + (1 << 16)]]][:, None])
                r2 = (d * d).sum(-1)
                s6 = (sig2 / r2) ** 3
                total += float((eps4 * (s6 * s6 - s6) + qq / r2.sqrt()).sum())
        return total

    def step(self, m: int, x: np.ndarray, uniform) -> float:
        """The Metropolis test of molecule m at x; returns the accepted dE."""
        de = self.molecule(m, x) - self.molecule(m, self.pos[m])
        if de < 0 or math.exp(-de / self.kT) >= uniform():
            self.pos[m] = x
            self.accepted += 1
            return de
        return 0.0

    def reference_loop(self, seed: int, steps: int) -> float:
        """The reference's loop with the C library's rand()."""
        libc = ctypes.CDLL(None)
        libc.srand(ctypes.c_uint(seed))
        real = lambda lo, hi: (hi - lo) * (libc.rand() / 2147483647) + lo
        e, self.accepted = self.system(), 0
        for _ in range(steps):
            m = min(int(real(0, self.n)), self.n - 1)
            v = min(int(real(0, self.a)), self.a - 1)
            move = np.array([real(-self.max_t, self.max_t) for _ in range(3)])
            x = self.pos[m] - self.pos[m][v]
            for axis in range(3):
                th = math.radians(real(-self.max_r, self.max_r))
                i, j = ((1, 2), (2, 0), (0, 1))[axis]
                p, q = x[:, i].copy(), x[:, j].copy()
                x[:, i] = p * math.cos(th) + q * math.sin(th)
                x[:, j] = q * math.cos(th) - p * math.sin(th)
            x += self.pos[m][v] + move
            x += self.L * ((x[self.prim] < 0).astype(float) - (x[self.prim] > self.L))
            e += self.step(m, x, lambda: real(0.0, 1.0))
        return e

    def chain(self, seed: int, chain_id: int, steps: int) -> float:
        """Steps of a device-resident chain: Philox draws, a turn about a
        random axis through a random atom, a shift."""
        key = (seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF)
        e, self.accepted = self.system(), 0
        wrap = lambda x: x - self.L * np.floor(x[self.prim] / self.L)
        self.pos = np.stack([wrap(x) for x in self.pos])
        unit = lambda r: ((r >> 8) + 0.5) * 2.0 ** -24
        for k in range(steps):
            a, b, c = (_philox((k & 0xFFFFFFFF, k >> 32, chain_id, blk), key) for blk in range(3))
            m, v = (a[0] * self.n) >> 32, (a[1] * self.a) >> 32
            move = np.array([2 * self.max_t * unit(r) - self.max_t for r in (a[2], a[3], b[0])])
            z, phi = 2 * unit(b[1]) - 1, 2 * math.pi * unit(b[2])
            th = math.radians(2 * self.max_r * unit(b[3]) - self.max_r)
            s = math.sqrt(1 - z * z)
            ax = np.array([s * math.cos(phi), s * math.sin(phi), z])
            x = self.pos[m] - self.pos[m][v]
            x = (x * math.cos(th) + np.cross(ax, x) * math.sin(th) +
                 np.outer(x @ ax, ax) * (1 - math.cos(th)))
            e += self.step(m, wrap(x + self.pos[m][v] + move), lambda: unit(c[0]))
        return e

    def xyz(self) -> np.ndarray:
        return self.pos.reshape(-1, 3)


def _philox(c, k):
    """Philox4x32-10 (Salmon et al., SC'11)."""
    c, k = list(c), list(k)
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(p1 >> 32) ^ c[1] ^ k[0], p1 & 0xFFFFFFFF, (p0 >> 32) ^ c[3] ^ k[1], p0 & 0xFFFFFFFF]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return c


def exact(case: dict, seed: int):
    """run()'s outputs in plain 64-bit arithmetic.  None where that takes
    minutes in numpy: the flexible molecules' moves, volume moves (both need
    the whole system's energy many times over), and the large batches."""
    kind = case["kind"]
    if kind in ("npt", "served") or case.get("species") == "flex":
        return None
    if kind == "batch":
        if case["chains"] * (case["warm"] + case["steps"]) > 8000:
            return None
        boxes, seeds = _batch_boxes(case, seed)
        e, acc, xyz = [], [], []
        for c, b in enumerate(boxes):
            x = _Exact(b)
            e.append(x.chain(int(seeds[c]), c, case["warm"] + case["steps"]))
            acc.append(x.accepted)
            xyz.append(x.xyz())
        xyz = np.concatenate(xyz)
        return {"energy": np.array(e), "accepted": np.array(acc),
                "xyz": [xyz[:, k].copy() for k in range(3)]}
    ctx = M.Context(0) if kind in ("molecule", "host_loop", "system", "device_loop") else None
    if kind == "device_loop":
        if case["boxes"] * case["steps"] > 8000:
            return None
        boxes = [_box(ctx, case["species"], case["n_mol"], case["cutoff"], seed * 17 + i)
                 for i in range(min(case["boxes"], 4))]
        e, acc, xyz = [], [], []
        for i in range(case["boxes"]):
            x = _Exact(boxes[i % len(boxes)])
            e.append(x.reference_loop(seed % 65521 + i, case["steps"]))
            acc.append(x.accepted)
            xyz.append(x.xyz())
        return {"energy": np.array(e), "accepted": np.array(acc), "xyz": np.concatenate(xyz)}
    x = _Exact(_box(ctx, case["species"], case["n_mol"], case["cutoff"], seed))
    if kind == "molecule":
        m = int(seed) % case["n_mol"]
        return {"energy": np.asarray(x.molecule(m, x.pos[m]))}
    if kind in ("system", "static"):
        e = x.system()
        return {"energy": np.array([e]) if kind == "static" else np.asarray(e)}
    if kind == "host_loop":
        e = x.reference_loop(seed & 0xFFFF, case["steps"])
    else:
        e = x.chain(seed, 0, case["warm"] + case["steps"])
    return {"energy": np.asarray(e), "accepted": x.accepted, "xyz": x.xyz()}
