"""Populations and fields through the caller's arrays in place and through the
staged copies, bit for bit: edges of the transposition's tiles (32 nodes along
x, eight (y, z) pairs), both lattices, every storage, both parities, arrays that
were never touched before the call."""
import numpy as np
import pytest

import cases
import lbmpsm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,periodic", [((31, 3, 3), (1, 1, 1)), ((32, 7, 9), (1, 0, 1)), ((30, 6, 14), (0, 0, 0)),
                                        ((70, 33, 40), (1, 1, 0)), ((33, 17, 1), (1, 1, 1)), ((256, 40, 1), (0, 0, 1)),
                                        ((3, 3, 3), (1, 1, 1))])
@pytest.mark.parametrize("storage", ["fp64", "fp32", "fp16", "bf16"])
def test_in_place_and_staged_agree(n, periodic, storage, monkeypatch):
    dim = 2 if n[2] == 1 else 3
    c = cases.Case("io", dim, n, periodic, 0.7, (1e-5, 0.0, 0.0), 0, 2, Nlc=9)
    lats = []
    for staging in ("0", "1"):
        monkeypatch.setenv("LBMPSM_HOST_STAGING", staging)
        lats.append(lbmpsm.Lattice(**c.params(), storage=storage))
    assert not lats[1].host_direct
    rng = np.random.default_rng(n[0])
    shape = lats[0].local + (lats[0].q,)
    none = (np.zeros(0, np.int32), np.zeros((0, 3)), np.zeros((0, 3)), np.zeros((0, 3)), np.zeros(0))
    for parity in range(2):
        f = rng.uniform(0.02, 0.3, shape)
        back = []
        for lat in lats:
            lat.set_populations(f)
            back.append(lat.populations())
        assert np.array_equal(*back)
        if storage == "fp64":  # what was set comes back on every stored entry that streams in
            same = back[0] == f
            assert same[tuple(slice(2, -2) if d < dim and n[d] > 4 else slice(None) for d in range(3))].all() or min(n[:dim]) <= 4
        fields = []
        for lat in lats:
            lat.request_macro()
            lat.step(*none)
            fields.append([lat.export_fields(0.5, 2.0, 3.0, as_double=d) for d in (True, False)])
        for a, b in zip(*fields):
            for p, q in zip(a, b):
                assert np.array_equal(p, q)
        assert np.array_equal(lats[0].populations(), lats[1].populations())
