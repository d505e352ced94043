"""When the device works on a caller's host arrays in place: only where it can
reach host memory and every array of the call is aligned to its elements
(csrc/host_access.h, host compilable), and every call that does so asks."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lammps-lbm-psm_gb300", "csrc")


def test_in_place_needs_aligned_arrays(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "host_access_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC,
                    os.path.join(ROOT, "tests", "native", "host_access_check.cpp"), "-o", exe], check=True)
    rows = [r.split() for r in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n") if r]
    assert len(rows) == 32
    for element, off, answers in rows:
        ok = int(off) % int(element) == 0
        assert answers == ("11110" if ok else "00010"), (element, off)


@pytest.mark.parametrize("call", ["lbmpsm_export_fields", "lbmpsm_get_populations", "lbmpsm_set_populations",
                                  "step_impl"])
def test_every_call_asks(call):
    src = open(os.path.join(CSRC, "capi.cu")).read()
    body = re.search(r"\nint %s\(.*?\n}\n" % call, src, re.S).group(0)
    assert re.search(r"if \([^{]*in_place\(h->host_direct,", body)
    assert "if (h->host_direct" not in body
