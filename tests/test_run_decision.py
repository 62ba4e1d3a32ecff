"""CPU: what the decision at the end of a resident run's attempt is given.

Two threads of different warps take it (run_finish, csrc/common.cuh): one
writes the next dt into the block's shared control block while the other may
still have to read this attempt's. So the callers pass the attempt's dt as a
value read before the phase's barrier; an expression that reads the control
block in the call would be evaluated by each thread after it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "cubble_gb300", "csrc")


@pytest.mark.parametrize("source", ["step.cu", "step_mixed.cu"])
def test_the_decision_gets_a_dt_read_before_the_barrier(source):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    calls = list(re.finditer(r"run_finish<\w+>\(([^;{]*)", text))
    assert calls
    for call in calls:
        dt = call.group(1).split(",")[3].strip()
        assert re.fullmatch(r"\w+", dt), "dt is read in the call: " + dt
        read = text.rfind("const double %s = c->dt;" % dt, 0, call.start())
        barrier = text.rfind("run_barrier(", 0, call.start())
        assert 0 <= read < barrier, "no read of dt before the barrier"
