"""The integer additions of the FP64 collide (csrc/fixed_f64.cuh, host
compilable) against IEEE double arithmetic, bit for bit, on random nodes near
rest: ties, denormal velocities, exact rest states and non-finite
populations among them."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lammps-lbm-psm_gb300", "csrc")


def test_integer_additions_are_the_ieee_additions(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "fixed_f64_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-x", "c++", "-I", CSRC,
                    os.path.join(ROOT, "tests", "native", "fixed_f64_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    rows = re.findall(r"(\S+) in_range (\S+) different (\d+)", out)
    assert [r[0] for r in rows] == ["D3Q19", "D2Q9", "factors"]
    for name, share, different in rows:
        assert int(different) == 0, out
        assert float(share) > 0.8, out
