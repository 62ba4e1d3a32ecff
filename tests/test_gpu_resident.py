"""GPU: resident runs (every attempt of a stretch inside one
cooperative kernel) against the launch per phase that larger contexts take.

The same foam is run in a context of its own size (resident) and in one whose
capacity lies beyond the resident range; both evaluate the same expressions
and differ in the order of reductions only. Bars: equal step, attempt, search
and deletion counts, bubbles and pairs; FP64 forms within 1e-11 of each row's
maximum over 30 steps (the sums of ~10 terms per bubble differ by ~1e-15 of
the row, growing along the run; the trajectory bar against the oracle is
1e-9), the mixed form within 1e-6 (FP32 reductions)."""
import numpy as np
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads
from helpers import assert_rows_close, by_index, position_ulp

pytestmark = pytest.mark.gpu

BEYOND = 5000001  # the smallest capacity with a launch per phase

OPTIONS = {
    "gas": {},
    "settle": dict(use_gas_exchange=0, increment_path=0),
    "walls": dict(wall=(1, 1, 0), wall_drag=0.1),
    "flow": dict(use_flow=1, flow_lbb=(0.0, 0.0, 0.0), flow_tfr=(8.0, 8.0, 8.0),
                 flow_vel=(0.02, 0.01, 0.0)),
    "shear": dict(use_flow=1, shear_speed=0.05, wall=(0, 1, 0), wall_drag=0.1),
}


def both(n, dim, precision, options, **kw):
    out = []
    for cap in (n, BEYOND):
        args = dict(seed=300 + n, capacity=cap, pair_capacity=16 * n + 64 if cap > n else 0,
                    precision=precision, use_graph=1)
        args.update(OPTIONS[options])
        args.update(kw)
        cfg, st = workloads.foam(n, dim, 0.9 if dim == 2 else 0.8, **args)
        for k in ("use_gas_exchange", "increment_path"):
            if k in args:
                setattr(cfg, k, args[k])
        f = cb.GpuFoam(cfg)
        f.load_state(st)
        workloads.prepare(f)
        out.append(f)
    return out


# one bubble; less, exactly and more than a warp; more than a block's threads;
# a ragged size; more bubbles and pairs than the resident threads (two rounds);
# the sizes around the change to more blocks per SM
@pytest.mark.parametrize("n,dim,options", [
    (1, 2, "gas"), (31, 2, "gas"), (32, 3, "gas"), (33, 2, "settle"), (257, 3, "settle"),
    (4099, 3, "gas"), (4097, 3, "walls"), (3001, 3, "flow"), (2999, 2, "flow"),
    (5003, 3, "shear"), (5000, 2, "shear"), (100003, 2, "gas"), (90001, 3, "gas"),
    (200003, 3, "walls"), (210001, 3, "shear"), (400009, 2, "flow"), (300007, 3, "settle")])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_resident_matches_launch_per_phase(n, dim, options, precision):
    a, b = both(n, dim, precision, options)
    la = a.launch_count()
    ra, rb = a.integrate(30), b.integrate(30)
    # one launch per stretch between searches and deletions
    assert a.launch_count() - la < ra["attempts"] + 30 * ra["searches"]
    for k in ("steps", "attempts", "searches", "deleted", "count", "num_pairs"):
        assert ra[k] == rb[k], k
    sa, sb = by_index(a.get_state()), by_index(b.get_state())
    rows = ["x", "y", "z", "r", "dxdt", "dydt", "dzdt", "drdt", "path", "dxdto"]
    assert_rows_close(sa, sb, rows, 1e-6 if precision == 1 else 1e-11, "resident ",
                      floor=position_ulp(sb))


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_resident_deletions_and_stops(precision):
    """Deletions inside the stretch, single steps, and a stop on the clock:
    the run returns at each and goes on from there."""
    a, b = both(3000, 2, precision, "gas", rstd=0.3, rclip=(0.01, 2.0), min_rad=0.2)
    for f in (a, b):
        for _ in range(5):
            f.integrate(1)
    ta, tb = (f.integrate_until(400, time=0.02) for f in (a, b))
    assert ta["deleted"] > 0 and ta["time_integer"] + ta["time_fraction"] >= 0.02
    for k in ("steps", "attempts", "searches", "deleted", "count", "num_pairs"):
        assert ta[k] == tb[k], k
    sa, sb = a.get_state(), b.get_state()
    assert (sa["index"] == sb["index"]).all()
    assert_rows_close(sa, sb, ["x", "y", "r"], 1e-6 if precision == 1 else 1e-11, "resident ")


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("sizes", [(1, 700, 5003, 2048, 12001), (100, 40009, 1, 90007, 30000)])
@pytest.mark.parametrize("dim,options,kw", [
    (2, "gas", {}), (3, "walls", {}), (3, "flow", {}),
    (2, "gas", dict(rstd=0.3, rclip=(0.01, 2.0), min_rad=0.2)),
    (2, "gas", dict(rstd=0.3, rclip=(0.01, 2.0), min_rad=0.3, capacity=130000))])
def test_resident_batch_matches_batched_launches(dim, options, kw, sizes, precision):
    """A batch of small foams (resident: every foam its own blocks and loop)
    against the same batch with one foam's capacity beyond the resident
    total (the batched launches): the foams search, delete and finish at
    different attempts. The larger foams take the runs with more blocks per SM;
    capacities above 5 10^5 in all let short rounds alternate with attempts of
    all foams together."""
    reports, states, launches = [], [], []
    for beyond in (0, 1):
        items = []
        for f, n in enumerate(sizes):
            args = dict(seed=900 + f, kappa=0.01 * (f + 1), precision=precision, use_graph=1)
            args.update(OPTIONS[options])
            args.update(kw)
            if beyond and f == 3:
                args.update(capacity=6000001, pair_capacity=16 * n)
            items.append(workloads.foam(n, dim, 0.9 if dim == 2 else 0.8, **args))
        batch = cb.GpuFoamBatch([c for c, _ in items])
        for (_, st), f in zip(items, batch.foams):
            f.load_state(st)
            workloads.prepare(f)
        n0 = batch.launch_count()
        reports.append(batch.integrate(40))
        launches.append(batch.launch_count() - n0)
        states.append([by_index(f.get_state()) for f in batch.foams])
        batch.close()
    assert launches[0] < launches[1]
    for f in range(len(sizes)):
        for k in ("steps", "attempts", "searches", "deleted", "count", "num_pairs"):
            assert reports[0][f][k] == reports[1][f][k], (f, k)
        assert_rows_close(states[0][f], states[1][f], ["x", "y", "z", "r", "dxdt", "drdt", "path"],
                          1e-6 if precision == 1 else 1e-11, "batch ",
                          floor=position_ulp(states[1][f]))


def dense_cluster(n, dim, seed):
    """A crowd in one corner of a wide box: more than 24 bubbles per occupied
    cell, rows beyond the partner stash."""
    cfg, st = workloads.foam(n, dim, 0.9 if dim == 2 else 0.8, seed=seed)
    rng = np.random.default_rng(seed)
    for k in "xyz"[:dim]:
        st[k][: n // 2] = 2.0 + rng.uniform(0.0, 4.0, n // 2)
    return cfg, st


# one to a few cells per axis (box sides from ~4 to ~100 units), walls, wide
# cells (24 and more bubbles each), rows that outgrow their stash, odd sizes
@pytest.mark.parametrize("n,dim,kind", [
    (1, 2, "plain"), (2, 3, "plain"), (40, 2, "plain"), (60, 3, "plain"), (200, 3, "plain"),
    (700, 3, "walls"), (2501, 2, "walls"), (5000, 3, "plain"), (9999, 2, "plain"),
    (4001, 3, "wide"), (3001, 2, "wide"), (900, 3, "cluster"), (800, 2, "cluster"),
    (50001, 3, "plain"), (99991, 2, "plain")])
@pytest.mark.parametrize("precision", [0, 1])
def test_resident_search_matches_launch_per_phase(n, dim, kind, precision):
    """One cooperative launch against a launch per phase: every row, the pair
    list and the neighbour counts bit for bit."""
    got = []
    for cap in (n, 100001):  # the smallest capacity with a launch per phase
        if kind == "cluster":
            cfg, st = dense_cluster(n, dim, 17)
        else:
            cfg, st = workloads.foam(n, dim, 0.9 if dim == 2 else 0.8, seed=50 + n,
                                     rstd=0.15, rclip=(0.3, 2.5),
                                     wall=(1, 0, 1) if kind == "walls" else (0, 0, 0))
        rng = np.random.default_rng(n)
        for k in ("dxdt", "drdto", "path", "error"):
            st[k] = rng.uniform(0.0, 1.0, n).astype(np.float32).astype(np.float64)
        cfg.capacity, cfg.precision, cfg.pair_capacity = cap, precision, 400 * n + 100
        f = cb.GpuFoam(cfg)
        f.load_state(st)
        if kind == "wide":
            f.set_tuning(cell_scale=3.5)
        for _ in range(2):  # the second one starts from a searched state
            f.search_neighbors()
        got.append((f.report(), f.get_state(), f.pairs()))
        f.close()
    (ra, sa, pa), (rb, sb, pb) = got
    assert ra["searches"] == rb["searches"] == 2 and ra["num_pairs"] == rb["num_pairs"]
    if kind == "cluster":
        assert np.bincount(pa[0], minlength=1).max() > (32 if dim == 3 else 16)
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
    assert np.array_equal(pa[0], pb[0]) and np.array_equal(pa[1], pb[1])


def test_resident_search_reports_a_full_pair_list():
    """A pair list too small stops the run at the search that finds it, with
    runs enqueued behind it."""
    cfg, st = workloads.foam(3000, 2, 0.9, seed=12, use_graph=1, pair_capacity=20000)
    probe = cb.GpuFoam(cfg)
    probe.load_state(st)
    probe.search_neighbors()
    first = probe.report()["num_pairs"]
    probe.close()
    cfg.pair_capacity = first + 5  # the foam relaxes into more listed pairs
    f = cb.GpuFoam(cfg)
    f.load_state(st)
    workloads.prepare(f)
    with pytest.raises(cb.CubbleError) as e:
        f.integrate(3000)
    assert e.value.code == 3
    r = f.report()
    assert r["status"] == 3 and 0 < r["steps"] < 3000
