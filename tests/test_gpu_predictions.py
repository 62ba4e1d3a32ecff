"""GPU: one attempt of the FP64 forms where the prediction lies outside the
ordinary range, against the FP64 oracle."""
import numpy as np
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads
from helpers import assert_rows_close, by_index

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


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("row", ["dxdto", "dydt", "drdto"])
def test_a_nan_that_enters_through_the_prediction(row, dim, precision):
    """A NaN in a previous rate reaches the prediction alone: non-finite, and
    not a step error that rejects until the cap."""
    cfg, st = lattice(dim, 18.0)
    st[row] = np.zeros(len(st["r"]))
    st[row][5] = np.nan
    for single in (False, True):
        g = cb.GpuFoam(workloads.sweep_config_as(cfg, precision=precision))
        g.load_state(st)
        g.search_neighbors()
        with pytest.raises(cb.CubbleError) as e:
            g.attempt() if single else g.integrate(1)
        assert e.value.code == 5, e.value


ROWS = ["xp", "yp", "rp", "dxdtp", "dydtp", "drdtp", "overlap"]


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("at", [3.0, -40.0, 1e9])
def test_bubbles_far_beyond_a_wall(oracle_mod, at, dim, precision):
    """Three bubbles lie many boxes beyond a wall, two of them overlapping, one
    moving: its step error rejects the first attempts, the pair moves apart,
    and the move since the search is seen."""
    cfg, st = lattice(dim, 18.0, wall=(1, 0, 0), wall_drag=0.1)
    n = len(st["r"])
    st["x"][:3] = at * 18.0 + np.array([0.0, 1.5, 60.0])
    for k in "yz"[:dim - 1]:
        st[k][:3] = 5.0
    st["dxdt"] = np.zeros(n)
    st["dxdt"][2] = 0.9  # error ~ h v: 4.5e-5 at the first dt
    g, o = both(oracle_mod, cfg, st, precision)
    assert np.array_equal(g.get_state()["index"], o.get_state()["index"])
    g.set_pairs(*o.pairs())  # the search's FP32 filter is for the box's surroundings
    a, b = g.attempt(), o.attempt()
    tol = max(1e-12, 8 * 2.0 ** -53 * abs(at) * 18.0)  # of rows of about 1
    rows = ROWS + (["zp", "dzdtp"] if dim == 3 else [])
    assert_rows_close(a, b, rows, tol, "far ")
    assert b["max_error"] > 1e-5
    place = 4 * np.spacing(abs(at) * 18.0 + 60.0)
    for k in ("error", "path_new"):
        assert np.max(np.abs(a[k] - b[k])) <= max(place, 1e-15), k
    for k in ("max_error", "max_expansion"):
        assert a[k] == pytest.approx(b[k], rel=1e-11, abs=place), k
    if abs(at) > 1e6:
        return  # the coordinates no longer resolve the tolerance
    rg, ro = g.integrate(4), o.integrate(4)
    for k in ("steps", "attempts", "searches", "count", "num_pairs"):
        assert rg[k] == ro[k], k
    sg, so = by_index(g.get_state()), by_index(o.get_state())
    assert_rows_close(sg, so, ["x", "y", "r", "dxdt", "path"], 1e-10, "far ")


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim,options", [
    (2, {}), (3, {}), (2, dict(wall=(1, 1, 0), wall_drag=0.2)),
    (3, dict(use_flow=1, flow_lbb=(0.0,) * 3, flow_tfr=(8.0,) * 3, flow_vel=(0.02, 0.01, 0.03))),
    (3, dict(use_flow=1, shear_speed=0.05, wall=(0, 0, 1), wall_drag=0.1))])
@pytest.mark.parametrize("dt", [40.0, 200.0, 2e4])
def test_a_step_far_too_large(oracle_mod, dt, dim, options, precision):
    """dt so large that some or all predictions leave the box, by up to many
    times its size: the attempt is that of the oracle, and rejected. Its
    positions reach ~10^4, so the forces carry ~10^-12 / d: 1e-9 of each row."""
    cfg, st = workloads.foam(1500, dim, 0.9 if dim == 2 else 0.8, seed=88, **options)
    g = cb.GpuFoam(workloads.sweep_config_as(cfg, precision=precision))
    o = oracle_mod.OracleFoam(cfg)
    for f in (g, o):
        f.load_state(st)
        workloads.prepare(f)
        f.integrate(3)
    s = o.get_state()  # the same rows for both
    g.load_state(s)
    o.load_state(s)
    for f in (g, o):
        f.search_neighbors()
        f.set_time(dt)
    a, b = g.attempt(), o.attempt()
    assert b["max_error"] > cfg.tfr[0] / 2
    rows = ROWS + (["zp", "dzdtp"] if dim == 3 else [])
    assert_rows_close(a, b, rows + ["error", "path_new"], 1e-9, "large step ")
    for k in ("max_error", "max_expansion", "total_overlap_area", "total_area"):
        assert a[k] == pytest.approx(b[k], rel=1e-9), k
    assert g.report()["time_step"] == o.report()["time_step"] == dt * 0.37


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("options", [{}, dict(wall=(1, 0, 0), wall_drag=0.1)])
def test_radii_in_a_wide_box(oracle_mod, dim, options, precision):
    """A radius keeps the bits of its double in a box 2^20 of it wide, where the
    unit of the positions is 2^-41: positions that are multiples of 2^-20 leave
    the radii as the only source of rounding. Bar: the oracle's own, ~1e-15 of
    each term (6e-16 R^2 for the overlap), ten times that through the mean-field
    difference of nearly equal 1/r."""
    cfg, st = lattice(dim, 18.0, **options)
    side = 2.0 ** 20
    cfg.tfr = cb._abi.D3(side, side, side if dim == 3 else 0.0)
    rng = np.random.default_rng(5)
    n = len(st["r"])
    for k in "xyz"[:dim]:
        st[k] = np.round(st[k] * 2.0 ** 20) / 2.0 ** 20
    for k in "yz"[:dim - 1]:
        st[k] = st[k] + 2.0 ** 18
    st["x"] = st["x"] + (0.0 if options else 2.0 ** 18)
    st["r"] = rng.uniform(0.9, 1.1, n)
    g, o = both(oracle_mod, cfg, st, precision)
    g.set_pairs(*o.pairs())
    a, b = g.attempt(), o.attempt()
    assert np.count_nonzero(b["overlap"]) > n / 2
    rows = ["dxdtp", "drdtp", "rp", "overlap"]
    assert_rows_close(a, b, rows, 2e-14, "wide box ")
    for k in ("total_overlap_area", "total_overlap_area_per_radius", "total_area"):
        assert a[k] == pytest.approx(b[k], rel=2e-14), k
    # the radius error |predicted - corrected|, beside no motion along y
    i = np.argmax(b["error"])
    assert abs(a["error"][i] - b["error"][i]) <= 2 * np.spacing(2.0 ** 18)


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("options", [{}, dict(wall=(1, 1, 0), wall_drag=0.1, use_flow=1,
                                              flow_lbb=(0.0,) * 3, flow_tfr=(9.0,) * 3,
                                              flow_vel=(0.02, 0.01, 0.0))])
def test_a_radius_beyond_what_the_search_saw(oracle_mod, dim, options, precision):
    """A bubble that grows to ten times the largest radius of the last search in
    one prediction leaves the radii's range, which that search sets. Bar: its
    own overlaps and area, of ~10^2, dominate the sums: 1e-13 of each row."""
    cfg, st = lattice(dim, 18.0, **options)
    n = len(st["r"])
    st["drdt"] = np.zeros(n)
    st["drdt"][4] = 6e4
    g, o = both(oracle_mod, cfg, st, precision)
    a, b = g.attempt(), o.attempt()
    i = int(np.flatnonzero(o.get_state()["index"] == 4)[0])
    assert b["error"][i] > 3.0 and b["overlap"][i] > 0.0
    rows = ["dxdtp", "dydtp", "drdtp", "rp", "overlap", "error"]
    assert_rows_close(a, b, rows, 1e-13, "grown ")
    for k in ("total_overlap_area", "total_area", "max_error", "total_volume_new"):
        assert a[k] == pytest.approx(b[k], rel=1e-13), k


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("dim", [2, 3])
def test_overlaps_of_bubbles_much_smaller_than_their_partner(dim, precision):
    """Bubbles of 2^-4 ... 2^-14 of their one partner's radius, inside it or cut
    by its surface, against exact rational arithmetic. Bar: a contained bubble's
    area to 4 roundings of FP64; of a cut one the rounding of (r2^2 - r1^2 + d^2),
    2^-53 R^2 a term, against r R: 2^-50 R / r."""
    from fractions import Fraction as F

    cfg, st = lattice(dim, 18.0, min_rad=0.0)
    n = len(st["r"])
    rng = np.random.default_rng(8)
    at = np.arange(6) * 3.0 + 1.0
    grid = np.meshgrid(*([at] * dim), indexing="ij")
    big = {k: g.ravel() for k, g in zip("xyz", grid)}
    small = np.round(2.0 ** -(4 + np.arange(n) % 11) * rng.uniform(1.0, 1.9, n) * 2.0 ** 40) / 2.0 ** 40
    inside = np.arange(n) // 11 % 2 == 0
    d = np.where(inside, 0.3, np.sqrt(1.0 + small ** 2 * rng.uniform(0.05, 0.5, n)))
    d = np.round(d * 2.0 ** 44) / 2.0 ** 44  # from a box face at 0: exact sums
    st = {"x": np.concatenate([big["x"], big["x"] + d]), "r": np.concatenate([np.ones(n), small])}
    for k in "yz":
        st[k] = np.tile(big.get(k, np.zeros(n)), 2)
    cfg.capacity, cfg.pair_capacity = 2 * n, 64 * n
    g = cb.GpuFoam(workloads.sweep_config_as(cfg, precision=precision))
    g.load_state(st)
    g.search_neighbors()
    a, s = g.attempt(), g.get_state()
    row = np.argsort(s["index"])
    for i in range(n):
        r = F(float(st["r"][n + i]))
        m = (F(float(st["x"][n + i])) - F(float(st["x"][i]))) ** 2
        if inside[i]:
            q, bar = r * r, 4 * 2.0 ** -53
        else:
            assert m > 1 and m < (1 + r) ** 2
            q, bar = r * r - (r * r - 1 + m) ** 2 / (4 * m), 2.0 ** -50 / float(r)
        want = np.pi * float(q) if dim == 3 else 2.0 * np.sqrt(float(q))
        got = a["overlap"][row[n + i]]
        assert abs(got - want) <= bar * want, (i, inside[i], float(r), got, want)
