"""Steps with images held in place run without the map once it changes
nothing: run_fixed, groups and the drag sensitivities against the same number
of ordinary steps, bit for bit, from a table that particles have just moved
over, with overlapping boxes and nodes claimed by three particles."""
import numpy as np
import pytest

import cases
import lbmpsm

pytestmark = pytest.mark.gpu


def _sets(case):
    """The case's images before and after its particles have moved."""
    tag, x, v, w, r = cases.initial_particles(case)
    out = []
    for k in range(2):
        out.append(cases.images(case, tag, x + 6.0 * k * v, v, w, r, cases.product_make_ghosts))
    return out


def _step(lat, g):
    return lat.step(g["tag"], g["x"], g["v"], g["omega"], g["radius"])


@pytest.mark.parametrize("name", ["dense_periodic_3d", "shear_3d", "dense_periodic_2d", "c2_sphere_3d", "closedbox_3d"])
@pytest.mark.parametrize("storage", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("nsteps", [1, 3, 4, 5, 9])
def test_run_fixed_equals_steps(name, storage, nsteps):
    case = cases.CASES[name]
    a, b = (cases.GpuBackend(case, storage, collide_tuning="default").lat for _ in range(2))
    first, moved = _sets(case)
    if len(first["tag"]) != len(moved["tag"]):
        first = moved
    for lat in (a, b):
        for g in (first, moved):
            _step(lat, g)
            lat.apply_bc()
    a.run_fixed(nsteps)
    for _ in range(nsteps):
        want = _step(b, moved)
        b.apply_bc()
    for p, q in zip(a.read_forces(len(moved["tag"])), want):
        assert np.array_equal(p, q)
    assert np.array_equal(a.populations(), b.populations())
    for p, q in zip(a.particle_table(), b.particle_table()):
        assert np.array_equal(p, q)


@pytest.mark.parametrize("nsteps", [3, 9, 14])
def test_group_equals_steps(nsteps):
    names = ["dense_periodic_3d", "c2_sphere_3d"]
    lats = [[cases.GpuBackend(cases.CASES[n], "fp32", collide_tuning="default").lat for n in names] for _ in range(2)]
    sets = [_sets(cases.CASES[n])[1] for n in names]
    for side in lats:
        for lat, g in zip(side, sets):
            _step(lat, g)
    grp = lbmpsm.Group(lats[0])
    grp.run_fixed(nsteps)
    for a, b, g in zip(*lats, sets):
        for _ in range(nsteps):
            want = _step(b, g)
        for p, q in zip(a.read_forces(len(g["tag"])), want):
            assert np.array_equal(p, q)
        assert np.array_equal(a.populations(), b.populations())
    grp.close()


def test_adjoint_and_tangent_end_where_steps_end():
    case = cases.CASES["c2_sphere_3d"]
    lats = [cases.GpuBackend(case, "fp64").lat for _ in range(3)]
    g = _sets(case)[0]
    im = (g["tag"], g["x"], np.zeros_like(g["v"]), g["omega"], g["radius"])
    got = lats[0].adjoint_drag(*im, 7, 2, 7, checkpoint_every=3)
    J, dJ = lats[1].tangent_drag(*im, 7, 2, 7, dtau=1.0)
    drag = []
    for _ in range(7):
        fh = lats[2].step(*im)[0]
        drag.append(fh[:, 0].sum())
    assert np.allclose(got["drag"], drag, rtol=1e-12, atol=0)
    assert J == got["J"] and abs(dJ - got["dtau"]) <= 1e-9 * abs(dJ)
    for lat in lats[:2]:
        assert np.array_equal(lat.populations(), lats[2].populations())
