"""GPU: deletion marks. The correct kernels write a mark only where a bubble
is to be deleted, unless the last attempt left marks behind; every attempt's
delete_flags must still be that attempt's alone."""
import numpy as np
import pytest

import cubble_gb300 as cb
from cubble_gb300 import workloads

pytestmark = pytest.mark.gpu


def foam(n, dim, precision, small, capacity):
    cfg, st = workloads.foam(n, dim, 0.8, rstd=0.1, seed=31, min_rad=0.2, precision=precision,
                             capacity=capacity)
    st["r"][:small] = 0.05
    return cfg, st


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim", [2, 3])
def test_marks_of_attempts_that_are_not_accepted(dim, precision):
    cfg, st = foam(700, dim, precision, 40, 1500)
    g = cb.GpuFoam(cfg)
    g.load_state(st)
    workloads.prepare(g)
    small = g.get_state(rows=("r",))["r"] < 0.2
    for _ in range(2):  # the second attempt follows one that left its marks
        a = g.attempt()
        assert np.array_equal(a["delete_flags"] != 0, small)
        assert a["num_to_be_deleted"] == 40
    g.profile_kernels(1)
    assert np.array_equal(g.attempt()["delete_flags"] != 0, small)
    # another state in the same context: fewer bubbles, then more, none to delete
    for n in (300, 1400):
        _, other = foam(n, dim, precision, 0, 1500)
        g.load_state(other)
        workloads.prepare(g)
        a = g.attempt()
        assert not a["delete_flags"].any() and a["num_to_be_deleted"] == 0
    # and a deletion after all of that removes its own bubbles only
    g.load_state(st)
    workloads.prepare(g)
    r = g.integrate(1)
    assert r["deleted"] == 40 and r["count"] == 660
    r = g.integrate(3)
    assert r["deleted"] == 40
    g.close()
