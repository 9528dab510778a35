"""Zeros, constants and sparse lines in the fixed-point line transform of the FP64
form (vk_fix.cuh), and the mean of its rounding errors, on the host."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LENGTHS = [8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768]


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("fix") / "fix_zero_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "vonkarman_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fix_zero_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    rows = {}
    for line in out.splitlines():
        f = line.split()
        rows.setdefault((f[0], int(f[1]), int(f[2])), []).append(f[3:])
    return rows


@pytest.mark.parametrize("length", LENGTHS)
def test_zero_operands_stay_zero(report, length):
    # a single entry, a constant and an empty line need no rounding: every
    # output, and the part that holds only zeros, is exact
    for inv in (0, 1):
        for kind, wrong in report[("zeros", length, inv)]:
            assert int(wrong) == 0, (inv, kind)


@pytest.mark.parametrize("length", LENGTHS)
def test_sparse_lines_keep_the_norm(report, length):
    # one real entry, real lines, constants of two sizes, a constant with a small
    # disturbance: one unit in the last place of the norm, as for dense lines
    for inv in (0, 1):
        for kind, err in report[("sparse", length, inv)]:
            assert float(err) < 2.0 ** -52, (inv, kind)


@pytest.mark.parametrize("length", LENGTHS)
def test_mean_error(report, length):
    # Output 0, whose errors would add up over the lines of a grid, has none.
    # Elsewhere the short components of quarter turns leave 1/16 of a unit and
    # those of twelfth turns 1/32: one butterfly meets at most one quarter turn
    # without a factor 3 in the length (1/16, and as much again from the stage
    # before), and 9/32 with one (its other stages less than 1/16).  Five standard errors of
    # the mean over 40000 lines, of a deviation below 1.8 units, are 0.045.
    for inv in (0, 1):
        (zero, worst), = report[("mean", length, inv)]
        assert float(zero) < 0.045
        assert float(worst) < (0.125 if length % 3 else 11.0 / 32.0) + 0.045
