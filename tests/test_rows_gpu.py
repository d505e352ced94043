"""The FP32 / FP16 / BF16 collide over row lengths: several short rows to a
tile (with a plane's last tile partly filled), one row, long rows in chunks,
rows too long or too few for the pipeline, on periodic and walled axes -- the
pipeline of every lattice against the direct kernel.  Long rows agree bit for
bit; shorter ones to FP32 rounding (their multiply-adds contract differently),
which two steps of a flow with moving particles keep below 2e-6 relative."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

SIZES = {
    "short_rows": (9, 30, 420),       # 28 rows a tile, the last two left over
    "rows_of_33": (33, 37, 330),      # seven rows of pitch 40, a remainder of two
    "rows_of_64": (64, 66, 140),
    "rows_of_128": (128, 33, 120),
    "rows_of_129": (129, 20, 20),
    "one_row": (256, 16, 16),
    "long_257": (257, 40, 34),
    "long_513": (513, 36, 36),
    "long_760": (760, 36, 36),
    "few_long_rows": (300, 20, 16),
    "long_2d": (603, 1300, 1),
}


@pytest.mark.parametrize("name", list(SIZES))
@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (0, 0, 0), (1, 0, 1)])
def test_pipeline_against_direct_kernel(name, storage, periodic, monkeypatch):
    n = SIZES[name]
    dim = 2 if n[2] == 1 else 3
    if dim == 2:
        periodic = periodic[:2] + (1,)
    r = min(5.0, min(n[:dim]) / 2.0 - 2.5)
    c = cases.Case("rows", dim, n, periodic, 0.7, (1e-6, 0.0, 0.0), 0, 4, Nlc=9, diam=(2 * r, 2 * r),
                   centres=[[n[0] / 2 + 0.3, n[1] / 2 - 0.2, n[2] / 2 + 0.1 if dim == 3 else 0.0],
                            [r + 2.6, n[1] / 2 - 0.4, n[2] / 2 + 0.2 if dim == 3 else 0.0]][:1 if n[0] < 30 else 2],
                   vel=0.02, spin=0.01, seed=n[0])
    lats = []
    for stages in (None, "0"):
        monkeypatch.delenv("LBMPSM_PIPE_STAGES", raising=False)
        if stages is not None:
            monkeypatch.setenv("LBMPSM_PIPE_STAGES", stages)
        lats.append(cases.GpuBackend(c, storage).lat)
    assert lats[1].info.collide_stages == 0
    tag, x, v, w, rr = cases.initial_particles(c)
    exact = n[0] > 256
    for _ in range(c.steps):
        g = cases.images(c, tag, x, v, w, rr, cases.product_make_ghosts)
        outs = [lat.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"]) for lat in lats]
        if exact:
            for a, b in zip(*outs):
                assert np.array_equal(a, b)
        x = cases.advance(c, x, v)
    fa, fb = (lat.populations() for lat in lats)
    if exact:
        assert np.array_equal(fa, fb)
    elif storage == "fp32":
        assert np.abs(fa - fb).max() <= 2e-6 * np.abs(fb).max()
    else:  # one unit in the last place of the stored deviation (11 or 8 bits) where FP32 rounds apart
        dev = np.abs(fb).max() * 0.1
        assert np.abs(fa - fb).max() <= dev * (2.0 ** -10 if storage == "fp16" else 2.0 ** -7)
    assert np.isfinite(fa).all()
