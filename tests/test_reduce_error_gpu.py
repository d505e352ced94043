"""Error of the FP64 forces, torques and stresslets against the exact sums of the
oracle's node forces: no larger (rms over many particles, relative to each
vector's largest component) than with every node's term scaled on its own and
the terms summed by 128 threads in strides, then by a butterfly and in the order
of the warps (the plain reduction, restated here)."""
import math
from fractions import Fraction

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def exact(parts, factor):
    """The sum of the doubles in parts, times factor, to 2^-106."""
    s = math.fsum(parts)
    return Fraction(s) * Fraction(factor) + Fraction(math.fsum(list(parts) + [-s])) * Fraction(factor)


def products(a, b):
    """a*b as two arrays of doubles with the exact products for sums (Dekker)."""
    p = a * b

    def split(x):
        t = 134217729.0 * x
        h = t - (t - x)
        return h, x - h
    ah, al = split(a)
    bh, bl = split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def plain(terms, where):
    """The plain reduction: thread where % 128 adds its terms in order."""
    acc = np.zeros(128)
    np.add.at(acc, where % 128, terms)
    total = 0.0
    for w in range(4):
        v = acc[32 * w:32 * w + 32]
        for o in (16, 8, 4, 2, 1):
            v = v + v[np.arange(32) ^ o]
        total += v[0]
    return total


@pytest.mark.parametrize("dim,n,count,diam", [(3, (64, 48, 56), 40, (8.0, 14.0)), (2, (300, 220, 1), 40, (10.0, 40.0))])
def test_error_of_the_sums(dim, n, count, diam):
    c = cases.Case("err", dim, n, (1, 1, 1), 0.7, (1e-5, 2e-5, 0.0), 0, 3, Nlc=9, diam=diam, seed=dim)
    rng = np.random.default_rng(dim)
    margin = np.array([diam[1] / 2 + 4] * dim + [0.0] * (3 - dim))
    x, r = cases.rsa(rng, count, diam, margin, np.array(n, float) * (np.arange(3) < dim) - margin, dim, 0.5)
    v = rng.normal(0.0, 0.03, x.shape) * (np.arange(3) < dim)
    w = rng.normal(0.0, 0.005, x.shape) * (1 if dim == 3 else np.arange(3) == 2)
    tag = np.arange(1, len(x) + 1, dtype=np.int32)
    gpu, orc = cases.GpuBackend(c, "fp64"), cases.OracleBackend(c)
    info = gpu.lat.info
    ff, tf = info.forceFactor, info.torqueFactor
    err = {k: ([], []) for k in "FTS"}
    for _ in range(c.steps):
        out = gpu.step(tag, x, v, w, r)
        orc.step(tag, x, v, w, r)
        ids, _, _, nodeF = orc.sim.pdata()
        for p in range(len(x)):
            got = np.concatenate([o[p] for o in out])
            slot = np.where(ids[..., 0] == tag[p], 0, np.where(ids[..., 1] == tag[p], 1, -1))
            i, j, k = np.nonzero(slot >= 0)
            order = np.lexsort((i, j, k))  # x fastest
            i, j, k = i[order], j[order], k[order]
            F = np.take_along_axis(nodeF[i, j, k].reshape(-1, 2, 3), slot[i, j, k][:, None, None], 1)[:, 0].T
            local = x[p] / c.dx + 1.0
            if dim == 2:
                local[2] = x[p, 2] / c.dx + 1.0
            d = [q - l for q, l in zip((i.astype(float), j.astype(float), k.astype(float)), local)]
            where = ((k - k.min()) * (np.ptp(j) + 1) + j - j.min()) * (np.ptp(i) + 1) + i - i.min()
            cross = [(1, 2), (2, 0), (0, 1)]
            pairs = [(1, 0), (2, 0), (2, 1)]
            ref, old = [], []
            for a in range(3):
                ref.append(exact(list(F[a]), ff))
                old.append(plain(F[a] * ff, where))
            for a, b in cross:
                parts = [*products(d[a], F[b]), *[-q for q in products(d[b], F[a])]]
                ref.append(exact(list(np.concatenate(parts)), tf))
                old.append(plain((d[a] * F[b] - d[b] * F[a]) * tf, where))
            for a in range(3):
                ref.append(-exact(list(np.concatenate(products(d[a], F[a]))), tf))
                old.append(-plain(d[a] * F[a] * tf, where))
            for a, b in pairs:
                parts = [*products(d[a], F[b]), *products(d[b], F[a])]
                ref.append(-exact(list(np.concatenate(parts)), tf) / 2)
                old.append(-plain(0.5 * (d[a] * F[b] + d[b] * F[a]) * tf, where))
            for name, sl in (("F", slice(0, 3)), ("T", slice(3, 6)), ("S", slice(6, 12))):
                scale = max(abs(float(q)) for q in ref[sl])
                for q, g, o in zip(ref[sl], got[sl], old[sl]):
                    err[name][0].append(float(abs(Fraction(float(g)) - q)) / scale)
                    err[name][1].append(float(abs(Fraction(float(o)) - q)) / scale)
    rms = {k: [float(np.sqrt(np.mean(np.square(e)))) for e in v] for k, v in err.items()}
    print(rms)
    for name, (here, before) in rms.items():
        assert here <= before, rms
