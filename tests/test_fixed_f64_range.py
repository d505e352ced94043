"""The range of the FP64 collide's integer path (csrc/fixed_f64.cuh): the lowest
density that the sums let through is what the header states, and equilibria and
differences there, at the largest velocities, are IEEE double arithmetic's."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lammps-lbm-psm_gb300", "csrc")


def test_lowest_densities(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "fixed_f64_range_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-x", "c++", "-I", CSRC,
                    os.path.join(ROOT, "tests", "native", "fixed_f64_range_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    rows = re.findall(r"(\S+) least_density (\S+) least_equilibrium (\S+) different (\d+)", out)
    assert [r[0] for r in rows] == ["D3Q19", "D2Q9"]
    for (name, density, equilibrium, different), low in zip(rows, (0.609375, 0.5546875)):
        assert int(different) == 0, out
        assert low <= float(density) < low * 1.001, out  # reached
        assert float(equilibrium) > 2.0 ** -7, out       # product62's lower limit
    header = open(os.path.join(CSRC, "fixed_f64.cuh")).read()
    assert "0.609375" in header and "0.5546875" in header
