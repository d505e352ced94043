"""The solid-fraction classification deals an image's rows to one block or to
several by the number of images: the FP64 table against the CPU oracle's with
numbers of images on both sides of the lines between one, several and sixteen
blocks (images of one particle are repeated, which leaves the table as it
is)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["dense_periodic_3d", "dense_periodic_2d"])
@pytest.mark.parametrize("n", [1, 151, 152, 284, 607, 608, 2500])
def test_table_with_many_images(name, n):
    case = cases.CASES[name]
    gpu, orc = cases.GpuBackend(case, "fp64"), cases.OracleBackend(case)
    tag, x, v, w, r = cases.initial_particles(case)
    mask = gpu.lat.stored_mask()
    for _ in range(2):
        g = cases.images(case, tag, x, v, w, r, cases.product_make_ghosts)
        k = np.arange(n) % len(g["tag"])
        a = [np.ascontiguousarray(np.asarray(g[f])[k]) for f in ("tag", "x", "v", "omega", "radius")]
        gpu.step(*a)
        orc.step(*a)
        for p, q in zip(gpu.lat.particle_table(), orc.sim.pdata()):
            assert np.array_equal(p[mask], q[mask])
        for _ in range(20):
            x = cases.advance(case, x, v)
