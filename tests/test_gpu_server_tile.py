"""The server runs jobs on the tile its caller chose: a job's energy is then the same
chain's in a batch of that tile to the last bit (the number of warps decides the order
of a step's FP32 sums), molecules of more than four atoms included."""
import numpy as np
import pytest

from mcgpu_gb300 import PREC_MIXED, ROT_AXIS, ChainBatch, Context, JobServer
from mcgpu_gb300.workloads import bicyclic_box, water_box
from test_gpu_fp64_items import CASES, mixed_box, one_primary

pytestmark = pytest.mark.gpu

ROUND = 50


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def jobs():
    return [bicyclic_box(500, cutoff=12.0, seed=3, lattice=True), water_box(400, seed=4),
            one_primary(mixed_box(*CASES["uneven_edges"])),
            one_primary(mixed_box(*CASES["one_species_5"]))]


@pytest.mark.parametrize("tile", [(64, 1, 0), (128, 1, 0), (256, 2, 0)])
def test_jobs_run_on_the_chosen_tile(ctx, tile):
    boxes = jobs()
    srv = JobServer(ctx, hbm_budget_bytes=64 << 20, max_slots=8, round_steps=ROUND, tile=tile)
    # isobaric, volume moves with FP32 pairs: both forms then start from the FP32 sums
    ids = [srv.submit(b, 100 + i, 8 * ROUND, chain_id=i, npt=True, pressure_atm=1.0,
                      max_dlnv=0.002, vol_precision=PREC_MIXED) for i, b in enumerate(boxes)]
    srv.drain()
    done = srv.results()
    srv.close()
    bt = ChainBatch(ctx, boxes, [100 + i for i in range(len(boxes))], rotation=ROT_AXIS)
    bt.set_tile(tile[0], tile[1], ROUND, tile[2])
    bt.set_npt(ROUND, 1.0, 0.002, PREC_MIXED)
    bt.run(8 * ROUND)
    for c, (i, s) in enumerate(zip(ids, bt.stats())):
        r = done[i].result
        assert r.energy == s.energy and r.accepted == s.accepted, c
        assert np.array_equal(done[i].coords,
                              np.stack(bt.download(c), 1)), c
    bt.close()
