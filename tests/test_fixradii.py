"""CPU: the FP64 form's pair terms with the radii in a finer unit than the
positions' (csrc/fixpair.cuh), compiled for the host from the same header. A
radius of 2^52 units or more, that is down to 2^-8 of the largest one a foam may
have, keeps every bit of its double, and the pair terms hold the bars of
test_fixpair.py (2^-50 for the deepest pairs' force, 2^-54 of R^2 for the
overlap) whatever the unit of the positions."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def found():
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = os.path.join(tempfile.mkdtemp(), "fixradii_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off",
                    os.path.join(HERE, "fixradii_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    return {ln.split()[0]: float(ln.split()[1]) for ln in out.splitlines() if ln.strip()}


def test_radii_are_exact(found):
    assert found["inexact"] == 0


def test_terms(found):
    assert found["count"] > 5e5 and found["refused"] == 0
    assert found["force"] <= 2.0 ** -50
    assert found["area"] <= 2.0 ** -54


def test_range(found):
    assert found["range"] == 0 and found["differ"] == 0
