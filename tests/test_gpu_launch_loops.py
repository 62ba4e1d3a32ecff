"""GPU: the loops that launch a kernel per phase, against the FP64 oracle and
the reference's golden vectors: the host's loop (use_graph 0), the graph with
its conditional nodes (use_graph 1), and both forms of the batched one. Contexts
of up to 5 10^6 bubbles and batches of up to 2 10^6 advance by resident runs
whatever use_graph says, so these tests take a capacity beyond that. Bars as in
test_gpu_parity.py, test_gpu_golden.py and test_gpu_batch.py."""
import numpy as np
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads
from cubble_gb300.foam import CubbleError
from helpers import assert_rows_close, by_index, position_ulp
from test_golden import FILES, config, ids, load, state
from test_gpu_batch import displacement_err
from test_gpu_golden import sorted_pairs
from test_gpu_parity import make

pytestmark = pytest.mark.gpu

BEYOND = 5000001        # the smallest capacity of a context with a launch per phase
BATCH_BEYOND = 2000001  # and of a batch

FLOW = dict(use_flow=1, flow_lbb=(0.0,) * 3, flow_tfr=(8.0,) * 3, flow_vel=(0.02, 0.01, 0.0))


def foam(case, oracle=None, precision=0, **over):
    """The foam beyond the limit and, on request, the oracle on the same state."""
    cfg, st = make(case, **over)
    n = len(st["x"])
    big = workloads.sweep_config_as(cfg, precision=precision, capacity=BEYOND,
                                    pair_capacity=16 * n + 64)
    out = [cb.GpuFoam(big)] + ([oracle.OracleFoam(cfg)] if oracle else [])
    for f in out:
        f.load_state(st)
        workloads.prepare(f)
    return out


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("case,over", [("2d", {}), ("3d", {}), ("3d-wallz", {}), ("2d", FLOW),
                                       ("3d-small", {})])
def test_trajectory(oracle_mod, case, over, precision, graph):
    g, o = foam(case, oracle_mod, precision, use_graph=graph, **over)
    n0 = g.launch_count()
    rg, ro = g.integrate(30), o.integrate(30)
    assert g.launch_count() - n0 >= 3 * rg["attempts"]  # a launch per phase
    for k in ("steps", "attempts", "searches", "deleted", "count", "num_pairs"):
        assert rg[k] == ro[k], k
    assert rg["time_step"] == pytest.approx(ro["time_step"], rel=1e-12)
    sg, so = by_index(g.get_state()), by_index(o.get_state())
    assert_rows_close(sg, so, ["x", "y", "z", "r", "dxdt", "dydt", "drdt", "path", "dxdto",
                               "error"], 1e-9, "trajectory ", floor=position_ulp(so))
    g.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", ["2d", "3d"])
def test_graph_matches_the_hosts_loop(case, precision):
    """Counts, states, and the graph's launch count."""
    (a,), (b,) = (foam(case, None, precision, use_graph=g) for g in (0, 1))
    la, lb = a.launch_count(), b.launch_count()
    ra, rb = a.integrate(40), b.integrate(40)
    for k in ("steps", "attempts", "searches", "deleted", "count"):
        assert ra[k] == rb[k], k
    sa, sb = by_index(a.get_state()), by_index(b.get_state())
    assert_rows_close(sa, sb, ["x", "y", "z", "r"], 1e-6 if precision else 1e-10, "graph ")
    assert b.launch_count() - lb == a.launch_count() - la > 0
    for f in (a, b):
        f.close()


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("path", FILES, ids=ids)
def test_deletion_matches_reference(path, graph):
    d = load(path)
    n = len(d["delete_in_x"])
    cfg = config(d, error_tolerance=1.0, skin_radius=1e9, time_step=1e-5, use_graph=graph,
                 capacity=BEYOND, pair_capacity=len(d["attempt_pi"]) + 16 * n)
    g = cb.GpuFoam(cfg)
    g.load_state(state(d, "delete_in_"))
    g.set_pairs(d["attempt_pi"], d["attempt_pj"])
    rep = g.integrate(1)
    assert rep["deleted"] == len(d["delete_out_to_be_deleted"])
    s = g.get_state()
    assert np.array_equal(s["index"], d["delete_out_index"])
    floor = position_ulp(state(d, "delete_in_"))
    for k in ("x", "y", "r", "dxdt", "drdt", "path", "error"):
        assert_rows_close({k: s[k]}, {k: d["delete_out_" + k]}, [k], 1e-12, floor=floor)
    i, j = g.pairs()
    assert np.array_equal(sorted_pairs(s, i, j), d["delete_out_pairs"])
    g.close()


@pytest.mark.parametrize("graph", [0, 1])
def test_reject_cap_and_single_steps(oracle_mod, graph):
    g, o = foam("2d", oracle_mod, 0, use_graph=graph)
    for _ in range(6):
        rg, ro = g.integrate(1), o.integrate(1)
        for k in ("steps", "attempts", "searches", "count", "num_pairs"):
            assert rg[k] == ro[k], k
    g.close()
    (g,) = foam("2d", None, 0, use_graph=graph, tol=1e-30, max_attempts=5)
    with pytest.raises(CubbleError) as e:
        g.integrate(1)
    assert e.value.code == 4 and g.report()["attempts"] == 5
    g.close()


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("kw", [{}, dict(rstd=0.3, rclip=(0.01, 2.0), min_rad=0.2)])
def test_batch_against_oracle(oracle_mod, kw, graph):
    """Three foams, with and without deletions, batched beyond the limit."""
    items = [workloads.foam(n, 2, 0.85, seed=50 + f, use_graph=graph, **kw)
             for f, n in enumerate((3000, 5200, 1800))]
    cfgs = [c for c, _ in items]
    cfgs[1] = workloads.sweep_config_as(cfgs[1], capacity=BATCH_BEYOND, pair_capacity=16 * 5200)
    batch = cb.GpuFoamBatch(cfgs)
    oracles = []
    for (cfg, st), bf in zip(items, batch.foams):
        o = oracle_mod.OracleFoam(cfg)
        for f in (bf, o):
            f.load_state(st)
            workloads.prepare(f)
        oracles.append(o)
    s0 = [by_index(bf.get_state()) for bf in batch.foams]
    n0 = batch.launch_count()
    reps = batch.integrate(10)
    assert batch.launch_count() - n0 >= 4 * max(r["attempts"] for r in reps)
    for f, ((cfg, _), bf, o) in enumerate(zip(items, batch.foams, oracles)):
        ro = o.integrate(10)
        for k in ("steps", "attempts", "searches", "deleted", "count", "num_pairs"):
            assert reps[f][k] == ro[k], (f, k)
        sb, so = by_index(bf.get_state()), by_index(o.get_state())
        assert np.array_equal(sb["index"], so["index"])
        if not kw:
            assert displacement_err(cfg, sb, so, s0[f]) <= 1e-11
        assert_rows_close(sb, so, ["x", "y", "r", "dxdt", "drdt"], 1e-9, "batch ")
        assert bf.total_volume() == pytest.approx(o.total_volume(), rel=1e-12)
    assert bool(kw) == (sum(r["deleted"] for r in reps) > 0)
    batch.close()
