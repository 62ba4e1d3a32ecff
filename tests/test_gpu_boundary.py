"""GPU: the flow and wall terms of the FP64 forms' correct kernel, which are
decided on fixed-point positions, against the FP64 oracle at the edges: faces
of the flow's box that cut bubbles, lie beyond the box or at infinity, an empty
box, walls on every axis, and a bubble with more neighbours than the table of
reciprocals has entries. Bar: 1e-11 of the row maximum (sums of up to ~150
neighbours in another order, 150 x 2^-53 each, and two accepted steps)."""
import numpy as np
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads
from helpers import assert_rows_close

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("low,high", [
    (0.2, 0.6), (0.0, 1.0), (-1e300, 1e300), (-INF, 0.5), (0.7, 0.3), (1.5, 2.5), (0.5, 0.5)])
@pytest.mark.parametrize("walls", [(0, 0, 0), (1, 1, 1)])
def test_boundary_terms(oracle_mod, low, high, walls, dim, precision):
    n = 2001
    wall = walls[:dim] + (0,) * (3 - dim)
    side = workloads.foam(n, dim, 0.8, seed=77)[0].tfr[0]
    at = lambda v: v * side if abs(v) < 1e6 else v  # noqa: E731
    args = dict(seed=77, wall=wall, wall_drag=0.3, use_flow=1, flow_lbb=(at(low),) * 3,
                flow_tfr=(at(high),) * 3, flow_vel=(0.02, -0.01, 0.03))
    cfg, st = workloads.foam(n, dim, 0.8, **args)
    st["r"][7] = 0.13 * side  # swallows its neighbours: more than 31
    cfg.pair_capacity = 40 * n
    out = []
    for f in (cb.GpuFoam(workloads.sweep_config_as(cfg, precision=precision)),
              oracle_mod.OracleFoam(cfg)):
        f.load_state(st)
        f.set_time(1e-5)
        f.search_neighbors()
        f.bootstrap()
        f.integrate(2)
        out.append((f.attempt(), f.get_state()))
    (ag, sg), (ao, so) = out
    assert so["num_neighbors"].max() > 31
    assert np.array_equal(sg["index"], so["index"])
    rows = ["dxdtp", "dydtp", "drdtp"] + (["dzdtp"] if dim == 3 else [])
    assert_rows_close(ag, ao, rows, 1e-11, "boundary ")
