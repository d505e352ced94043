"""The table update with moving particles whose tags are positive, negative,
or negative only from a later step on (a node's flag leaves such slots out):
the FP64 table against the CPU oracle's and the FP32 tags against it, every
step."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["dense_periodic_3d", "dense_periodic_2d"])
@pytest.mark.parametrize("negative_from", [0, 2, 99])
def test_slot_tags(name, negative_from):
    case = cases.CASES[name]
    gpu, low, orc = cases.GpuBackend(case, "fp64"), cases.GpuBackend(case, "fp32"), cases.OracleBackend(case)
    tag, x, v, w, r = cases.initial_particles(case)
    mask = gpu.lat.stored_mask()
    for step in range(5):
        g = cases.images(case, tag, x, v, w, r, cases.product_make_ghosts)
        t = np.array(g["tag"])
        if step >= negative_from:
            t = np.where(t % 2 == 0, -t, t).astype(t.dtype)
        for b in (gpu, low, orc):
            b.step(t, g["x"], g["v"], g["omega"], g["radius"])
        ids, eps, us = gpu.lat.particle_table()
        ids_o, eps_o, us_o, _ = orc.sim.pdata()
        assert np.array_equal(ids[mask], ids_o[mask])
        assert np.array_equal(eps[mask], eps_o[mask])
        assert np.array_equal(us[mask], us_o[mask])
        assert np.array_equal(low.lat.particle_table()[0][mask], ids_o[mask])
        for _ in range(20):
            x = cases.advance(case, x, v)
