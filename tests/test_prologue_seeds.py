"""The prologue's paths that start a Newton iteration from a float reciprocal,
on the CPU with that seed at both ends of its stated error (2^-21): wherever
they answer they give the exact chain's float."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.mark.parametrize("err", ["0x1p-21f", "-0x1p-21f"])
def test_seeds_at_the_edge_of_their_error(tmp_path, err):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "prologue_seed_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-DPF_SEED_ERR={err}",
                    "-I", os.path.join(ROOT, "simfast21_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "prologue_seed_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "4000000", "1"], capture_output=True, text=True, check=True).stdout
    rows = {r[0]: tuple(map(int, r[1:])) for r in map(str.split, out.splitlines()) if r[0] != "#"}
    for name, (n, bad, left) in rows.items():
        assert n > 0 and bad == 0, out
        assert left <= n / 2 ** 13, out  # one in 2^14 is left to the next path
    assert set(rows) == {"rrec", "xhi"}
