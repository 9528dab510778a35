"""The fixed-point line transform of the FP64 form (vk_fix.cuh) on the host:
every plan, forward and inverse, against a long double DFT."""

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
    exe = str(tmp_path_factory.mktemp("fix") / "fix_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "vonkarman_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fix_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    acc, bias = {}, {}
    for line in out.splitlines():
        f = line.split()
        if f[0] == "accuracy":
            acc[(int(f[1]), int(f[2]), int(f[3]))] = (float(f[4]), float(f[5]))
        else:
            bias[(int(f[1]), int(f[2]))] = (float(f[3]), float(f[4]))
    return acc, bias


@pytest.mark.parametrize("length", LENGTHS)
def test_error_below_one_ulp_of_the_norm_and_below_doubles(report, length):
    # one unit in the last place of a double relative to the line's norm (the
    # bound derived in vk_fix.cuh), and no more than an FFT in doubles, for
    # white, steep, exponential, single-mode and padded lines
    for inv in (0, 1):
        for kind in range(5):
            fix, dbl = report[0][(length, inv, kind)]
            assert fix < 2.0 ** -52, (inv, kind)
            assert fix <= dbl, (inv, kind)


@pytest.mark.parametrize("length", LENGTHS)
def test_rounding_bias_stays_below_half_a_quantum(report, length):
    # the mean error of every output over 1500 lines: short twiddles leave up to
    # 1/8 of a unit each and no output of a line meets more than two in a stage,
    # plus 5 standard errors of the mean
    for inv in (0, 1):
        worst, noise = report[1][(length, inv)]
        assert worst < 0.25 + 5.0 * noise
