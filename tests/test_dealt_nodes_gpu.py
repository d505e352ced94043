"""The FP64 collide deals a block's nodes to its threads by how many particles
hold them: against the CPU oracle, bit for bit, with blocks of nodes of two
particles, of one and of none, a last block that is not full, and a lattice of
one block."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,diam", [((11, 11, 1), 4.0), ((127, 17, 1), 9.0), ((129, 33, 1), 17.0),
                                    ((17, 18, 19), 8.0), ((33, 20, 21), 11.0), ((128, 16, 16), 9.0)])
def test_nodes_of_two_one_and_no_particles(n, diam):
    dim = 2 if n[2] == 1 else 3
    mid = [n[0] / 2 + 0.3, n[1] / 2 - 0.2, n[2] / 2 + 0.1 if dim == 3 else 0.0]
    gap = min(diam + 0.4, n[0] - diam - 2.0)  # shells that share nodes
    centres = [[mid[0] - gap / 2, mid[1], mid[2]], [mid[0] + gap / 2, mid[1], mid[2]]]
    c = cases.Case("dealt", dim, n, (1, 1, 1), 0.7, (1e-6, 0.0, 0.0), 0, 3, Nlc=6, diam=(diam, diam),
                   centres=centres, vel=0.02, spin=0.01, seed=n[0])
    gpu, orc = cases.GpuBackend(c, "fp64"), cases.OracleBackend(c)
    tag, x, v, w, r = cases.initial_particles(c)
    m = gpu.lat.stored_mask()
    for _ in range(c.steps):
        g = cases.images(c, tag, x, v, w, r, cases.product_make_ghosts)
        a = gpu.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])
        b = orc.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])
        assert np.array_equal(gpu.lat.populations()[m], orc.sim.populations()[m])
        scale = max(np.abs(b[0]).max(), 1e-300)
        assert np.abs(a[0] - b[0]).max() <= 1e-12 * scale
