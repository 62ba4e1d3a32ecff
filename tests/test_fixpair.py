"""CPU: the fixed-point pair terms of the FP64 form (csrc/fixpair.cuh),
compiled for the host from the same header, against long double arithmetic on
the same integers, in 2D and 3D, over box units, radius ratios up to 2^4,
overlaps from 10^-9 to the containment of one centre, and components of zero.

Bars, from the arithmetic: the two reciprocals carry 2^-54 each (a residual
in units 2^-53, rounded), at most 8 units of the pair's scale (d >= R / 8), the
products and the conversion 2^-54: below 2^-50 in the worst (deepest) pair, and
2^-53 of f0 r.m.s., the rounding of one FP64 operation; the overlap 2^-54 of
R^2 (products to 2^-56, the integers of the squares to 2^-58)."""
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
    d = tempfile.mkdtemp()
    exe = os.path.join(d, "fixpair_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off",
                    os.path.join(HERE, "fixpair_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    return {ln.split()[0]: float(ln.split()[1]) for ln in out.splitlines() if ln.strip()}


@pytest.mark.parametrize("dim", [2, 3])
def test_force_and_overlap(found, dim):
    assert found["force%d" % dim] <= 2.0 ** -50
    assert found["force_rms"] <= 2.0 ** -53
    assert found["area%d" % dim] <= 2.0 ** -54


def test_range(found):
    """No pair with d >= 0.14 R and positive radii is refused, every pair
    outside the range is, and the containment test is right up to rounding."""
    assert found["count"] > 1e6
    assert found["refused"] == 0
    assert found["taken_outside"] == 0
    assert found["inside"] == 0


def test_conversions(found):
    assert found["to_fixed"] <= 0.5
    assert found["round_trip"] == 0


def test_norm(found):
    """Norms of integer differences in float-float: 2^-45, as its root and
    squares, and no bias beyond the last place of a double."""
    assert found["norm"] <= 2.0 ** -45
    assert found["norm_bias"] <= 2.0 ** -52
