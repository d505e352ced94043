"""Long rows in 2-D: which kernel takes them (FP32: the direct one up to 750
stored nodes a row, and where the populations outgrow the L2 cache), and the same
bits from both."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,storage,pipeline", [
    ((750, 1300, 1), "fp32", False), ((751, 1300, 1), "fp32", True), ((900, 3700, 1), "fp32", False),
    ((600, 1300, 1), "fp16", True), ((900, 1300, 1), "bf16", True), ((900, 300, 1), "fp32", False)])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (0, 0, 1)])
def test_long_rows(n, storage, pipeline, periodic, monkeypatch):
    c = cases.Case("rows2d", 2, n, periodic, 0.7, (1e-6, 2e-6, 0.0), 0, 3, Nlc=9, diam=(9.0, 9.0),
                   centres=[[n[0] / 2 + 0.3, n[1] / 2 - 0.2, 0.0], [7.6, 20.3, 0.0]], vel=0.03, spin=0.01, seed=n[0])
    monkeypatch.delenv("LBMPSM_PIPE_STAGES", raising=False)
    a = cases.GpuBackend(c, storage)
    monkeypatch.setenv("LBMPSM_PIPE_STAGES", "0")
    b = cases.GpuBackend(c, storage)
    if n[0] == 750:  # walls store a node more at either end
        pipeline = a.lat.info.storage_dims[0] > 750
        assert pipeline == (not periodic[0])
    assert (a.lat.info.collide_stages > 0) == pipeline and b.lat.info.collide_stages == 0
    tag, x, v, w, r = cases.initial_particles(c)
    for _ in range(c.steps):
        g = cases.images(c, tag, x, v, w, r, cases.product_make_ghosts)
        for p, q in zip(*[s.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"]) for s in (a, b)]):
            assert np.array_equal(p, q)
        x = cases.advance(c, x, v)
    assert np.array_equal(a.lat.populations(), b.lat.populations())
