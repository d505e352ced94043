"""The FP64 collide with a body force along each axis, along two, and out of the
plane of a 2-D lattice (u_z = F_z/(2 rho) and its part of the Guo term are the
reference's: src/LBM_PSM_dynamics.h:102-116), against the CPU oracle, bit for
bit: near rest, where the integer units form the sums, and far from it."""
import numpy as np
import pytest

import cases
from test_collide_f64_gpu import state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(33, 18, 1), (17, 18, 19)])
@pytest.mark.parametrize("speed", [0.0, 0.02, 0.2])
@pytest.mark.parametrize("force", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (0, -1, 1), (1, 1, 1)])
@pytest.mark.parametrize("particle", [False, True])
def test_populations_bit_for_bit(n, speed, force, particle):
    dim = 2 if n[2] == 1 else 3
    c = cases.Case("axes", dim, n, (1, 1, 1), 0.7, tuple(3e-4 * f for f in force), 0, 3, Nlc=6, diam=(5.0, 5.0),
                   centres=[[n[0] / 2 + 0.3, n[1] / 2 - 0.2, n[2] / 2 + 0.1 if dim == 3 else 0.0]],
                   vel=0.5 * speed, spin=0.01, seed=n[0])
    gpu, orc = cases.GpuBackend(c, "fp64"), cases.OracleBackend(c)
    f = state(np.random.default_rng([n[0], int(1000 * speed)]), gpu.lat.local, dim, speed, 0.01)
    gpu.lat.set_populations(f)
    orc.sim.set_populations(f)
    tag, x, v, w, r = cases.initial_particles(c)
    k = slice(None) if particle else slice(0)
    m = gpu.lat.stored_mask()
    for _ in range(c.steps):
        g = cases.images(c, tag[k], x[k], v[k], w[k], r[k], cases.product_make_ghosts)
        gpu.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])
        orc.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])
        assert np.array_equal(gpu.lat.populations()[m], orc.sim.populations()[m])
