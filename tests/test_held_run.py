"""The order of a group's steps, of its questions whether the tables have
settled and of its timings of the two plans (csrc/held_run.h, host compilable),
on a model of the group: tables that settle with the first to sixth map or never,
runs of every length, errors of every call."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lammps-lbm-psm_gb300", "csrc")


def test_plans_are_timed_on_like_steps(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "held_run_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC,
                    os.path.join(ROOT, "tests", "native", "held_run_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok "), out.stdout
