"""Populations set from an array that nothing has touched yet (its pages are not
there): no slower than through a staging copy, in which the host takes those
page faults.  The device's own cost 15 us a page: ten times the staged call for
an array of 80 MB."""
import time

import numpy as np
import pytest

import cases
import lbmpsm

pytestmark = pytest.mark.gpu


def test_untouched_zeros(monkeypatch):
    c = cases.Case("zeros", 3, (96, 80, 70), (1, 1, 1), 0.7, (0.0, 0.0, 0.0), 0, 1, Nlc=9)
    t = {}
    for staging in ("0", "1"):
        monkeypatch.setenv("LBMPSM_HOST_STAGING", staging)
        lat = lbmpsm.Lattice(**c.params())
        if staging == "0" and not lat.host_direct:
            pytest.skip("host memory is not coherent: every call stages")
        best = 1e9
        for _ in range(5):
            f = np.zeros(lat.local + (lat.q,))
            lat.synchronize()
            t0 = time.perf_counter()
            lat.set_populations(f)
            best = min(best, time.perf_counter() - t0)
        t[staging] = best
        assert not lat.populations().any()
    assert t["0"] < 2 * t["1"], t
