"""The rigid device loop (k_plain_rigid: moves drawn and staged ahead, hits
pooled over the CTA) where it can go wrong: one molecule (every accepted move
is followed by one of the same molecule, staged again), two, more than one
segment of 512 candidates, molecules of 1 to 64 atoms, more steps than one
launch takes (the generator's state carried over) -- against the host loop on
the same rand() stream.

The same draws and FP64 pair terms in another order: equal decisions, energies
within 1e-9 of the larger end's, coordinates within 1e-9 A (the device's
and the C library's sines differ by an ulp a step)."""
import numpy as np
import pytest

from mcgpu_gb300 import PREC_FP64, PREC_MIXED, Context, GpuBox
from mcgpu_gb300.workloads import water_box
from test_gpu_fp64_items import mixed_box

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def boxes(kind):
    if kind == "one":
        return mixed_box(3, 1, (5,), (24.0, 24.0, 24.0), 9.0)
    if kind == "two":
        return mixed_box(4, 2, (3, 7), (20.0, 22.0, 24.0), 8.0)
    if kind == "lengths":
        return mixed_box(5, 70, (1, 64, 2, 16, 3), (30.0, 33.0, 36.0), 9.0)
    box = water_box(kind)
    box.cutoff = min(box.cutoff, 0.5 * float(box.size[0]))
    return box


@pytest.mark.parametrize("kind,steps", [("one", 300), ("two", 4300), ("lengths", 300),
                                        (33, 300), (513, 300), (1100, 100)])
def test_rigid_device_loop_equals_host_loop(ctx, kind, steps):
    box = boxes(kind)
    g, h = GpuBox(ctx, box, PREC_FP64), GpuBox(ctx, box, PREC_FP64)
    d = g.run_plain_device(77, steps)
    r = h.run_plain_native(77, steps)
    assert (d.accepted, d.rejected) == (r.accepted, r.rejected)
    scale = max(1.0, abs(r.energy0), abs(r.energy))
    assert abs(d.energy0 - r.energy0) <= 1e-9 * scale
    assert abs(d.energy - r.energy) <= 1e-9 * scale
    assert np.abs(np.stack(g.download()) - np.stack(h.download())).max() <= 1e-9
    g.close()
    h.close()


@pytest.mark.parametrize("n_mol", [33, 513])
def test_rigid_device_loop_fp32_pairs(ctx, n_mol):
    """FP32 pairs: the running energy against a fresh sum of the final box, within
    1e-5 of the larger of the two ends' energies."""
    g = GpuBox(ctx, boxes(n_mol), PREC_MIXED)
    d = g.run_plain_device(78, 400)
    assert d.accepted + d.rejected == 400
    e = g.system_energy()
    assert abs(d.energy - e) <= 1e-5 * max(1.0, abs(e), abs(d.energy0))
    g.close()
