"""GPU: resident runs (small contexts: every attempt of a stretch inside one
cooperative kernel) against the launch per phase that larger contexts take.

The same foam is run in a context of its own size (resident) and in one whose
capacity lies beyond the resident range; both evaluate the same expressions
and differ in the order of reductions only. Bars: equal step, attempt, search
and deletion counts, bubbles and pairs; FP64 forms within 1e-11 of each row's
maximum over 30 steps (the sums of ~10 terms per bubble differ by ~1e-15 of
the row, growing along the run; the trajectory bar against the oracle is
1e-9), the mixed form within 1e-6 (FP32 reductions)."""
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads
from helpers import assert_rows_close, by_index, position_ulp

pytestmark = pytest.mark.gpu

BEYOND = {2: 600001, 3: 400001}  # the smallest capacity with a launch per phase

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
    for cap in (n, BEYOND[dim]):
        args = dict(seed=300 + n, capacity=cap, pair_capacity=16 * BEYOND[dim] if cap > n else 0,
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
# a ragged size; more bubbles and pairs than the resident threads (two rounds)
@pytest.mark.parametrize("n,dim,options", [
    (1, 2, "gas"), (31, 2, "gas"), (32, 3, "gas"), (33, 2, "settle"), (257, 3, "settle"),
    (4099, 3, "gas"), (4097, 3, "walls"), (3001, 3, "flow"), (2999, 2, "flow"),
    (5003, 3, "shear"), (5000, 2, "shear"), (100003, 2, "gas"), (90001, 3, "gas")])
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
@pytest.mark.parametrize("dim,options,kw", [
    (2, "gas", {}), (3, "walls", {}), (3, "flow", {}),
    (2, "gas", dict(rstd=0.3, rclip=(0.01, 2.0), min_rad=0.2))])
def test_resident_batch_matches_batched_launches(dim, options, kw, precision):
    """A batch of small foams (resident: every foam its own blocks and loop)
    against the same batch with one foam's capacity beyond the resident
    total (the batched launches): the foams search, delete and finish at
    different attempts."""
    sizes = (1, 700, 5003, 2048, 12001)
    reports, states, launches = [], [], []
    for beyond in (0, 1):
        items = []
        for f, n in enumerate(sizes):
            args = dict(seed=900 + f, kappa=0.01 * (f + 1), precision=precision, use_graph=1)
            if beyond and f == 3:
                args.update(capacity=1000001, pair_capacity=16 * n)
            args.update(OPTIONS[options])
            args.update(kw)
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
