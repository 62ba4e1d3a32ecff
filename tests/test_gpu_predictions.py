"""GPU: one attempt of the FP64 forms where the prediction lies outside the
ordinary range, against the FP64 oracle."""
import numpy as np
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads
from helpers import assert_rows_close

pytestmark = pytest.mark.gpu


def lattice(dim, side, **kw):
    """Bubbles of radius 1 three apart in a periodic box, every other pair
    along x pushed together until it overlaps."""
    at = np.arange(6) * (side / 6.0)
    grid = np.meshgrid(*([at] * dim), indexing="ij")
    st = {k: g.ravel() + 0.7 for k, g in zip("xyz", grid)}
    n = len(st["x"])
    st["x"] = st["x"] + np.where(np.arange(n) // 6 ** (dim - 1) % 2 == 0, 0.6, -0.6)
    st.setdefault("z", np.zeros(n))
    st["r"] = np.ones(n)
    st["index"] = np.arange(n, dtype=np.int32)
    cfg, _ = workloads.foam(n, dim, 0.5, seed=3, **kw)
    cfg.lbb = cb._abi.D3(0.0, 0.0, 0.0)
    cfg.tfr = cb._abi.D3(side, side, side if dim == 3 else 0.0)
    return cfg, st


def both(oracle_mod, cfg, st, precision):
    g = cb.GpuFoam(workloads.sweep_config_as(cfg, precision=precision))
    o = oracle_mod.OracleFoam(cfg)
    for f in (g, o):
        f.load_state(st)
        f.search_neighbors()
    return g, o


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim", [2, 3])
def test_a_predicted_radius_below_zero(oracle_mod, dim, precision):
    """A bubble that shrinks so fast that its prediction is negative (0.5 -
    0.6): the area of the mean-field term is the signed one in 2D. Bar: rp
    cancels to a tenth (6 x 2^-53), 1/rp^2 triples that, 1e-13 in all."""
    cfg, st = lattice(dim, 18.0, min_rad=0.01)
    n = len(st["r"])
    st["r"][4] = 0.5
    st["drdt"] = np.zeros(n)
    st["drdt"][4] = -4000.0
    g, o = both(oracle_mod, cfg, st, precision)
    a, b = g.attempt(), o.attempt()
    assert b["total_overlap_area"] > 0
    assert_rows_close(a, b, ["drdtp", "rp", "error", "dxdtp", "overlap"], 1e-13, "below zero ")
    for k in ("total_area", "total_area_per_radius", "total_volume_new", "max_error"):
        assert a[k] == pytest.approx(b[k], rel=1e-13), k
    assert np.array_equal(a["delete_flags"], b["delete_flags"])
