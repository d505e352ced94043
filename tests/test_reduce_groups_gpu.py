"""Reduction of images of more row groups than are held at a time (64: above
about 44 nodes of diameter for FP64 spheres, 510 for FP64 discs, 70 for FP32
spheres), by the eight blocks of a cluster and by one block (more images than
multiprocessors), and of images whose later blocks of the cluster have no row.

From rest, with the image in translation, each node's force has the image's
velocity for direction, so the terms of a force component share one sign and
their sum in any order is within n*2^-53 of the exact one (n nodes), relative:
twice that between two orders.  Torque and stresslet terms are such forces
times at most the radius, two of them a node."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def image(c, diam, copies):
    """The case's one particle and copies of a small one in a far corner."""
    x = np.array([c.centres[0]] + [[3.5, 3.5, 3.5 if c.dim == 3 else 0.0]] * copies)
    v = np.zeros_like(x)
    v[0] = (0.02, -0.015, 0.01 if c.dim == 3 else 0.0)
    r = np.array([diam / 2] + [1.5] * copies)
    tag = np.array([1] + [2] * copies, np.int32)
    return tag, x, v, np.zeros_like(x), r


@pytest.mark.parametrize("dim,n,diam,storage", [
    (3, (72, 72, 72), 60.0, "fp64"),
    (3, (62, 62, 62), 60.0, "fp64"),    # box as wide as the period: every node of it is visited
    (2, (540, 540, 1), 520.0, "fp64"),
    (3, (88, 88, 88), 76.0, "fp32"),
    (3, (24, 24, 24), 2.0, "fp64"),     # one group: seven blocks without a row
    (3, (24, 24, 24), 2.0, "fp32"),
])
def test_large_images(dim, n, diam, storage):
    c = cases.Case("groups", dim, n, (1, 1, 1), 0.7, (0.0, 0.0, 0.0), 0, 1, Nlc=9, diam=(diam, diam),
                   centres=[[n[0] / 2 + 0.3, n[1] / 2 - 0.2, n[2] / 2 + 0.1 if dim == 3 else 0.0]])
    a = image(c, diam, 0)
    few = cases.GpuBackend(c, storage).step(*a)
    if (3.5 + 1.5 + 3.0 - n[0] / 2) * (3 if dim == 3 else 2) ** 0.5 < -diam / 2 - 3.0:
        # more images than multiprocessors: one block an image, the same sums
        many = cases.GpuBackend(c, storage).step(*image(c, diam, 400))
        for p, q in zip(few, many):
            assert np.array_equal(p[0], q[0])
    if storage == "fp64":
        ref = cases.OracleBackend(c).step(*a)
        nodes = np.pi / 4 * (diam + 2) ** 2 if dim == 2 else np.pi / 6 * (diam + 2) ** 3
        F = np.abs(ref[0][0]).max()
        assert F > 0
        assert np.abs(few[0][0] - ref[0][0]).max() <= 2 * nodes * U * F
        for p, q in zip(few[1:], ref[1:]):
            assert np.abs(p[0] - q[0]).max() <= 2 * nodes * U * 2 * (diam / 2 + 2) * F
