"""Host arrays that are not aligned to their elements (a packed file read into a
buffer): the same results as aligned ones, which the device works on in place
where it can."""
import numpy as np
import pytest

import cases
import lbmpsm

pytestmark = pytest.mark.gpu


def unaligned(a, off):
    """A copy of array a that starts off bytes into its buffer."""
    buf = np.zeros(a.nbytes + 32, np.uint8)
    first = (-buf.ctypes.data) % 16 + off
    v = buf[first:first + a.nbytes].view(a.dtype).reshape(a.shape)
    v[...] = a
    assert v.ctypes.data % 16 == off
    return v


def lattice():
    c = cases.Case("una", 3, (21, 18, 34), (1, 1, 1), 0.7, (1e-5, 0.0, 0.0), 0, 2, Nlc=9)
    return lbmpsm.Lattice(**c.params())


NONE = (np.zeros(0, np.int32), np.zeros((0, 3)), np.zeros((0, 3)), np.zeros((0, 3)), np.zeros(0))


@pytest.mark.parametrize("off", [1, 4, 8, 12])
def test_populations(off):
    a, b = lattice(), lattice()
    f = np.random.default_rng(off).uniform(0.02, 0.3, a.local + (a.q,))
    a.set_populations(f)
    b.set_populations(unaligned(f, off))
    want = a.populations()
    assert np.array_equal(want, b.populations())
    got = unaligned(np.zeros_like(f), off)
    b._check(b.lib.lbmpsm_get_populations(b.h, got.ctypes.data_as(lbmpsm._D)))
    assert np.array_equal(want, got)


@pytest.mark.parametrize("off", [1, 2, 4, 8, 12])
@pytest.mark.parametrize("as_double", [True, False])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_fields(off, as_double, which):
    a = lattice()
    a.request_macro()
    a.step(*NONE)
    want = a.export_fields(0.5, 2.0, 3.0, as_double=as_double)
    got = [np.zeros_like(w) for w in want]
    got[which] = unaligned(got[which], off)
    a._check(a.lib.lbmpsm_export_fields(a.h, int(as_double), 0.5, 2.0, 3.0, *[g.ctypes.data for g in got]))
    for p, q in zip(want, got):
        assert np.array_equal(p, q)


@pytest.mark.parametrize("storage", ["fp64", "fp32"])
@pytest.mark.parametrize("which", range(6))
def test_step(storage, which):
    """Image arrays and outputs at odd offsets, some steps aligned in between."""
    c = cases.CASES["shear_3d"]
    a, b = cases.GpuBackend(c, storage).lat, cases.GpuBackend(c, storage).lat
    tag, x, v, w, r = cases.initial_particles(c)
    for step in range(8):
        g = cases.images(c, tag, x, v, w, r, cases.product_make_ghosts)
        arrays = [np.ascontiguousarray(g[k]) for k in ("tag", "x", "v", "omega", "radius")]
        want = a.step(*arrays)
        out = np.empty(12 * len(arrays[0]))
        if step not in (1, 5):
            if which < 5:
                arrays[which] = unaligned(arrays[which], 2 if which == 0 else 4)
            else:
                out = unaligned(out, 4)
        got = b.step(*arrays, out=out)
        for p, q in zip(want, got):
            assert np.array_equal(p, q)
        assert np.array_equal(a.populations(), b.populations())
        x = cases.advance(c, x, v)
