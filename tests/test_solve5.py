"""The refined FP32 solve of the local Newton's 5x5 systems
(csrc/local_solve.cuh) has the accuracy of an FP64 solve rounded to FP32: both
are compared with the same FP32 system solved in long double, over slip slopes
from far below the elastic stiffness to a billion times it."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path_factory.mktemp("solve5") / "solve5_check")
    # no contraction: the compensated products rely on each rounding
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + inc,
                    "-I" + os.path.join(REPO, "m-themes_gb300", "csrc"), os.path.join(HERE, "solve5_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe, "20000"], check=True, capture_output=True, text=True).stdout
    return [[float(t) for t in line.split()] for line in out.splitlines()]


def test_error_is_that_of_a_rounded_fp64_solve(rows):
    for dec, n, taken, worst, mean, worst64, mean64 in rows:
        # rounding each entry of x to FP32 leaves at most 1/2 ulp: 2^-24 |x_i|, so 1 in these
        # units; the refinement's own error is at most 2^-30 |x|
        assert worst <= 1.0 + 2.0 ** -6 and worst64 <= 1.0, (dec, worst, worst64)
        assert mean <= mean64 * (1.0 + 2.0 ** -6), (dec, mean, mean64)


def test_ordinary_systems_are_taken(rows):
    # slopes up to a hundred times the elastic compliance (the flow's own range) all take the
    # refined path; the rest is left to FP64
    assert all(r[2] >= 0.999 * r[1] for r in rows if r[0] <= -3)
