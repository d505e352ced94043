"""The FP64 collide against the CPU oracle, bit for bit, on states near rest
(sums on the integer units), far from it (FP64 sums) and across the border
between the two, with rows that are no multiple of a warp or a block, with and
without a body force, and a particle in the middle."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

W19 = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
W9 = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
E19 = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0),
                (-1, -1, 0), (1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0),
                (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1)], float)
E9 = np.array([(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0),
               (1, -1, 0)], float)


def state(rng, local, dim, speed, drho):
    E, w = (E9, W9) if dim == 2 else (E19, W19)
    u = rng.uniform(-speed, speed, tuple(local) + (3,))
    if dim == 2:
        u[..., 2] = 0.0
    u[rng.random(tuple(local)) < 0.1] = 0.0
    rho = 1.0 + rng.uniform(-drho, drho, tuple(local))
    eu = u @ E.T
    uu = (u * u).sum(-1)[..., None]
    f = w * rho[..., None] * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * uu)
    f *= 1.0 + rng.uniform(-0.01, 0.01, f.shape)
    for d in range(dim):  # periodic halo planes hold their twins
        idx = [slice(None)] * 4
        src = list(idx)
        idx[d], src[d] = 0, local[d] - 2
        f[tuple(idx)] = f[tuple(src)]
        idx[d], src[d] = local[d] - 1, 1
        f[tuple(idx)] = f[tuple(src)]
    return f


@pytest.mark.parametrize("n", [(33, 18, 1), (130, 16, 1), (17, 18, 19), (31, 16, 16), (129, 16, 16)])
@pytest.mark.parametrize("speed,drho", [(0.0, 0.0), (0.02, 0.01), (0.09, 0.13), (0.2, 0.3)])
@pytest.mark.parametrize("force", [0.0, 1e-5])
def test_populations_and_forces_bit_for_bit(n, speed, drho, force):
    dim = 2 if n[2] == 1 else 3
    c = cases.Case("f64", dim, n, (1, 1, 1), 0.7, (force, -0.5 * force, 0.0), 0, 3, Nlc=6, diam=(5.0, 5.0),
                   centres=[[n[0] / 2 + 0.3, n[1] / 2 - 0.2, n[2] / 2 + 0.1 if dim == 3 else 0.0]],
                   vel=0.5 * speed, spin=0.01, seed=n[0])
    gpu, orc = cases.GpuBackend(c, "fp64"), cases.OracleBackend(c)
    f = state(np.random.default_rng([n[0], int(1000 * speed)]), gpu.lat.local, dim, speed, drho)
    gpu.lat.set_populations(f)
    orc.sim.set_populations(f)
    tag, x, v, w, r = cases.initial_particles(c)
    m = gpu.lat.stored_mask()
    for _ in range(c.steps):
        g = cases.images(c, tag, x, v, w, r, cases.product_make_ghosts)
        a = gpu.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])
        b = orc.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])
        assert np.array_equal(gpu.lat.populations()[m], orc.sim.populations()[m])
        scale = max(np.abs(b[0]).max(), 1e-300)
        assert np.abs(a[0] - b[0]).max() <= 1e-12 * scale
