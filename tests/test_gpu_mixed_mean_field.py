"""GPU: the mixed form's 2D sum of area over radius, a constant for every
bubble. The sum has to be the constant times their number, whatever the grid,
the knobs or the batch that computes it: the FP32 rounding of a sum over
threads and blocks (up to 10^-7) shifts every bubble's gas flux alike, so the
same foam would run apart with its context's capacity or its batch's tile."""
import numpy as np
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads

pytestmark = pytest.mark.gpu

CONSTANT = float(np.float32(2.0) * np.float32(np.pi))


@pytest.mark.parametrize("n,capacity,knobs", [
    (1000, 1000, {}), (10007, 10007, {}), (10007, 5000001, {}), (300001, 300001, {}),
    (10007, 5000001, dict(step_blocks=1)), (90001, 5000001, dict(step_blocks=2))])
def test_sum_of_area_over_radius(n, capacity, knobs):
    cfg, st = workloads.foam(n, 2, 0.9, seed=5, precision=1, capacity=capacity,
                             pair_capacity=16 * n + 64, use_graph=1)
    g = cb.GpuFoam(cfg)
    if knobs:
        g.set_tuning(**knobs)
    g.load_state(st)
    workloads.prepare(g)
    assert g.attempt()["total_area_per_radius"] == CONSTANT * n  # of the predict phase
    g.load_state(st)
    workloads.prepare(g)
    g.integrate(3)
    assert g.attempt()["total_area_per_radius"] == CONSTANT * n  # of an accepted attempt
    g.close()


def test_the_same_foam_in_batches_of_other_tiles():
    """One foam alone, in a batch of two, and in one with another tile and the
    batched launches: volumes within the rounding of FP32 sums in another order
    (10^-7 of a flux that changes the volume by 10^-5 over 60 steps; the
    constant's own rounding showed as 2 10^-9 over 300)."""
    cfg, st = workloads.foam(10007, 2, 0.9, seed=5, precision=1, use_graph=1)
    volumes = []
    for tile, extra in ((0, 0), (2048, 3000), (256, 3000), (8192, 2100000)):
        if not tile:
            foams = [cb.GpuFoam(cfg)]
            batch = None
        else:
            other, so = workloads.foam(3000, 2, 0.9, seed=6, precision=1, use_graph=1,
                                       capacity=extra, pair_capacity=64000)
            batch = cb.GpuFoamBatch([cfg, other])
            batch.set_tile(tile)
            foams = batch.foams
            foams[1].load_state(so)
            workloads.prepare(foams[1])
        foams[0].load_state(st)
        workloads.prepare(foams[0])
        (batch or foams[0]).integrate(60)
        volumes.append(foams[0].total_volume())
        (batch or foams[0]).close()
    assert np.ptp(volumes) <= 2e-11 * volumes[0], volumes
