"""LBMPSM_PIPE_STAGES takes the pipeline with that many stages, on lattices whose
tiles hold several short rows too, and the results are the same bit for bit
whatever the number (include/lbmpsm.h): rows of one and of several a tile, every
FP32-collision storage, moving spheres, walls and seams."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(20, 72, 72), (100, 72, 72), (20, 24, 16), (200, 40, 40), (129, 40, 40),
                               (192, 24, 30)])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (0, 0, 0)])
@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
def test_any_number_of_stages(n, periodic, storage, monkeypatch):
    c = cases.Case("stages", 3, n, periodic, 0.7, (1e-5, 2e-5, -1e-5), 0, 4, Nlc=9, nparts=12, diam=(5.0, 7.0),
                   vel=0.05, spin=0.01, seed=n[0])
    tag, x, v, w, r = cases.initial_particles(c)
    rng = np.random.default_rng(n[1])
    v, f0 = rng.normal(0.0, 0.05, v.shape), None  # (towards walls too)
    got = {}
    for stages in (2, 3, 4, 5):
        monkeypatch.setenv("LBMPSM_PIPE_STAGES", str(stages))
        b = cases.GpuBackend(c, storage)
        if f0 is None:
            f0 = b.lat.populations() * (1.0 + rng.uniform(-0.05, 0.05, b.lat.local + (b.lat.q,)))
        b.lat.set_populations(f0)
        g = cases.images(c, tag, x, v, w, r, cases.product_make_ghosts)
        F = [b.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])[0] for _ in range(c.steps)]
        assert b.lat.get_info().collide_stages == stages
        got[stages] = [b.lat.populations()] + F
    for stages in (2, 4, 5):
        for p, q in zip(got[stages], got[3]):
            assert np.array_equal(p, q), stages
