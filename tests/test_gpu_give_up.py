"""GPU: a barrier of a resident run or search that gives up.

The launch is cooperative, so every arrival comes; the waits are bounded all
the same. give_up_check.cu makes one run out (a grid that lacks a block) and
makes others end at once (an arrival count that says some block gave up): the
call must return CB_ERR_CUDA, nothing may be scattered with indexes that were
not published, and the context must work again once a state is loaded."""
import ctypes as C
import glob
import os
import subprocess
import tempfile

import numpy as np
import pytest

from cubble_gb300 import _abi, buildlib, workloads

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(gpu_lib):
    objects = sorted(glob.glob(os.path.join(buildlib.OUT, "*.cu.o")))
    if len(objects) != len(buildlib.sources()):
        buildlib.build(force=True)
        objects = sorted(glob.glob(os.path.join(buildlib.OUT, "*.cu.o")))
    so = os.path.join(tempfile.mkdtemp(), "give_up.so")
    subprocess.run([buildlib.nvcc()] + buildlib.NVCC_FLAGS +
                   ["-shared", os.path.join(HERE, "give_up_check.cu")] + objects + ["-o", so],
                   check=True)
    lib = C.CDLL(so)
    lib.give_up.argtypes = [C.POINTER(_abi.Config), C.POINTER(_abi.StateView)]
    return lib


@pytest.mark.parametrize("dim,precision", [(2, 0), (3, 0), (2, 1), (3, 1)])
def test_a_barrier_that_gives_up(checker, dim, precision):
    cfg, st = workloads.foam(3001, dim, 0.9 if dim == 2 else 0.8, seed=77, precision=precision)
    view = _abi.StateView()
    view.count = len(st["x"])
    keep = {k: np.ascontiguousarray(st[k], np.float64) for k in ("x", "y", "z", "r")}
    for k, a in keep.items():
        setattr(view, k, a.ctypes.data_as(_abi.PD))
    assert checker.give_up(C.byref(cfg), C.byref(view)) == 0
