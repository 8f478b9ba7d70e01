"""The neutral fraction's sum from chunk pairs (neutral_sum.h) against the
serial sum, on the CPU: boxes of one value, whose serial sum drifts away from
the exact one until it leaves a binade in another chunk (the first two at
1024^3, near 2^29 and 2^30), and boxes whose sum ends on a binade."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("neutral") / "neutral_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "simfast21_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "neutral_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("N, values", [(1024, ["0.2", "0.180400446", "0.00099845673"]),
                                       (128, ["0", "0.5", "0.75", "0.3", "0.9999999", "1", "1e-17"]),
                                       (24, ["0", "0.3"])])
def test_composed_sum_is_the_serial_sum(check, N, values):
    out = subprocess.run([check, str(N ** 3), *values], capture_output=True, text=True, check=True).stdout
    rows = [r.split() for r in out.strip().splitlines()]
    assert len(rows) == len(values)
    for x, got, want in rows:
        assert got == want, x


def test_terms_are_multiples_of_2_to_the_minus_53(check):
    """1.0 - x of the float x in [0, 1], in integers."""
    out = subprocess.run([check, "units", "20000"], capture_output=True, text=True, check=True).stdout.split()
    assert int(out[1]) > 2000000 and int(out[2]) == 0
