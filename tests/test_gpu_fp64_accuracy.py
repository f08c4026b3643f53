"""FP64 pair terms against their true values: the LJ term of a close pair multiplies a
relative error of the distance by twelve, so 1/r^2 and sigma_ab^2 must not carry more
of it than the reference's own FP64 arithmetic (SimulationStep.cpp:344-375: a square
root for sigma_ab, one for epsilon_ab, a division by r^2)."""
import numpy as np
import pytest

from mcgpu_gb300 import PREC_FP64, Context, GpuBox
from mcgpu_gb300.workloads import BoxData
from test_gpu_fp64_items import device_energy

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def pairs(seed: int, k: int) -> BoxData:
    """k^3 pairs of one-site molecules, pairs 14 A apart; r = 0.5 to 0.8 of sigma_ab.
    Coordinates are multiples of 2^-30, so that their differences are exact."""
    rng = np.random.default_rng(seed)
    n = k ** 3
    c = (np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * 14.0
    sig, eps = rng.uniform(1.0, 4.0, (n, 2)), rng.uniform(0.01, 0.3, (n, 2))
    d = rng.normal(size=(n, 3))
    d *= (rng.uniform(0.5, 0.8, n) * np.sqrt(sig[:, 0] * sig[:, 1]) /
          np.linalg.norm(d, axis=1))[:, None]
    xyz = np.stack([c, c + d], 1).reshape(-1, 3)
    xyz = np.round(xyz * 2.0 ** 30) / 2.0 ** 30
    one = np.arange(2 * n)
    return BoxData(x=xyz[:, 0].copy(), y=xyz[:, 1].copy(), z=xyz[:, 2].copy(), sigma=sig.ravel(),
                   epsilon=eps.ravel(), charge=np.zeros(2 * n), mol_start=one,
                   mol_len=np.ones(2 * n), mol_pidx_start=one, mol_pidx_count=np.ones(2 * n),
                   pidx=one, size=np.full(3, 14.0 * k), cutoff=5.0, temperature=300.0,
                   max_translate=0.1, max_rotate=1.0).normalise()


def lj(box, t, reference: bool):
    """Each pair's term in floating type t; reference: the reference's operations."""
    x = np.stack([box.x, box.y, box.z], 1).astype(t).reshape(-1, 2, 3)
    d = x[:, 1] - x[:, 0]
    r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
    s, e = (v.astype(t).reshape(-1, 2) for v in (box.sigma, box.epsilon))
    ss, eps = s[:, 0] * s[:, 1], np.sqrt(e[:, 0] * e[:, 1])
    if reference:
        ss = np.sqrt(ss) * np.sqrt(ss)
    s6 = (ss / r2) ** 2 * (ss / r2)
    return t(4) * eps * (s6 * s6 - s6)


def test_lj_terms_are_as_exact_as_the_reference_s(ctx):
    box = pairs(5, 10)
    true = lj(box, np.longdouble, False)
    g = GpuBox(ctx, box, PREC_FP64)
    got = np.array([g.mol_energy(2 * i, 0) for i in range(box.n_mol // 2)])
    g.close()
    err = lambda v: np.abs((v.astype(np.longdouble) - true) / true).astype(float)
    ref = err(lj(box, np.float64, True))
    print("mean relative error", err(got).mean(), "the reference's", ref.mean())
    assert err(got).mean() <= ref.mean()
    assert err(got).max() <= 60 * 2.0 ** -53      # 12 x (r2 3, 1/r2 1, sigma 1) roundings at most


def test_static_lj_terms_are_as_exact_as_the_reference_s(ctx):
    """The same for the energy over the caller's rows, pair by pair."""
    box = pairs(6, 6)
    true = lj(box, np.longdouble, False)
    got = []
    for i in range(box.n_mol // 2):
        b = box.copy()
        for k in ("x", "y", "z", "sigma", "epsilon", "charge"):
            setattr(b, k, getattr(box, k)[2 * i:2 * i + 2].copy())
        b.mol_start = b.mol_pidx_start = b.pidx = np.arange(2)
        b.mol_len = b.mol_pidx_count = np.ones(2)
        got.append(device_energy(b.normalise()))
    err = lambda v: np.abs((v.astype(np.longdouble) - true) / true).astype(float)
    ref = err(lj(box, np.float64, True))
    print("mean relative error", err(np.array(got)).mean(), "the reference's", ref.mean())
    assert err(np.array(got)).mean() <= ref.mean()
