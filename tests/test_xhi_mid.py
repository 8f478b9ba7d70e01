"""The residual neutral fraction's fast path up to ratios of one half, on the
CPU: where it answers it gives the exact chain's float, it answers for all but
one float in 2^16 (a guard band of 2^-41 around midpoints 2^-23 apart, with a
factor to spare), and from one half up it leaves every float to the chain."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.fixture(scope="module")
def octaves(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("xhi") / "xhi_mid_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "simfast21_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "xhi_mid_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    return {int(r[0]): tuple(map(int, r[1:])) for r in map(str.split, out.strip().splitlines())}


@pytest.mark.parametrize("e", [-5, -4, -3, -2, -1, 0])
def test_octave(octaves, e):
    n, bad, left = octaves[e]
    assert bad == 0
    if e == -5:  # the octave below: its own rule leaves more
        assert left < n
    else:
        assert left <= n / 2 ** 16 if e <= -2 else left == n
