"""The row count of shell nodes (solid_fraction.cuh shell_count), restated in
numpy FP32 operation for operation, against the reference's FP64 sub-cell
loop (src/LBM_PSM_exchangeParticleData.cpp:144-168).  The device's approximate
square root may be off by 2^-23 of its value, so the restatement pushes each
root up or down by as much; a row the rule calls certain must give the
reference's count either way, and an open row may have one open sub-cell."""
import numpy as np
import pytest

F32 = np.float32
U = F32(2.0 ** -24)
DELTA = np.array([-0.5 + (i + 0.5) * 0.1 for i in range(10)])
SUB = np.array([F32(-0.45) + F32(0.1) * F32(k) for k in range(10)], dtype=F32)
MAGIC = F32(12582912.0)


def fma(a, b, c):  # FP32 operands: the product is exact in FP64 and the sum rounds once more at most
    return F32(np.longdouble(a) * np.longdouble(b) + np.longdouble(c))


def row_rule(d, r, xl, node, dim, push):
    """Per row: (indices, count of the rule or None where open, open sub-cell)."""
    xi = np.floor(xl).astype(int)
    xf = (xl - xi).astype(F32)
    df = [F32(node[k] - xi[k]) - xf[k] for k in range(3)]
    rsq = F32(r * r)
    ax, ay, az = abs(df[0]), abs(df[1]), abs(df[2]) if dim == 3 else F32(-1)
    pc = 2 if az >= ax and az >= ay else (1 if ay >= ax else 0)
    pb = (1, 0, 1)[pc]
    pa = 3 - pc - pb
    dca, da, db = abs(df[pc]), df[pa], df[pb]
    ea, eb = abs(da) + F32(2), abs(db) + F32(2)
    m = F32(8) * U * ((ea * ea if dim == 3 else F32(0)) + eb * eb + rsq)
    eps = F32(10) * (m / (dca - F32(0.45))) + F32(2) * U * (F32(40) * dca + F32(200))
    if not dca >= F32(0.75) or not eps < F32(0.25):
        return None
    K, open_ = F32(0.5) - dca, F32(0.5) - eps
    rows = []
    for a in range(10 if dim == 3 else 1):
        ta = da + SUB[a]
        x = rsq - ta * ta if dim == 3 else rsq
        for b in range(10):
            tb = db + SUB[b]
            t = x - tb * tb
            h = F32(np.sqrt(t)) * (F32(1) + F32(push) * F32(2) * U) if t >= 0 else F32(np.nan)
            w = F32(0) if np.isnan(h) else min(max(h + K, F32(0)), F32(1))
            n = fma(w, F32(10), MAGIC) - MAGIC
            if abs(fma(w, F32(10), -n)) >= open_:
                rows.append((a, b, None, int(np.floor(w * F32(10)))))
            else:
                rows.append((a, b, int(n), None))
    return pa, pb, pc, df[pc] < 0, rows


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("rmax", [1.2, 3.0, 9.0, 60.0])
def test_rows_called_certain_hold_the_reference_count(dim, rmax):
    rng = np.random.default_rng([dim, int(rmax * 10)])
    half = np.sqrt(3.1 if dim == 3 else 2.1) / 2.0
    ruled = opened = 0
    for trial in range(220):
        r = rng.uniform(0.3, rmax)
        xl = rng.uniform(-30.0, 200.0, 3)
        if trial % 4 == 1:  # centres on nodes and sub-cell planes: many exact ties
            xl = np.round(xl * 20) / 20
            r = max(round(r * 20) / 20, 0.3)
        if dim == 2:
            xl[2] = 0.0
        dr = rng.normal(size=3)
        if dim == 2:
            dr[2] = 0.0
        dr /= np.linalg.norm(dr)
        node = np.round(xl + dr * (r + rng.uniform(-half, half))).astype(int)
        if dim == 2:
            node[2] = 0
        d = node - xl
        if trial % 4 == 2:  # a sub-cell centre a hair from the surface
            i = rng.integers(0, 10, 3)
            s2 = sum((d[k] + DELTA[i[k]]) ** 2 for k in range(dim))
            r = float(np.sqrt(s2)) * (1.0 + 1e-12 * rng.integers(-1, 2))
            if r < 0.3:
                continue
        got = row_rule(d, r, xl, node, dim, (-1, 0, 1)[trial % 3])
        if got is None:
            continue
        ruled += 1
        pa, pb, pc, flip, rows = got
        sq = [(d[k] + DELTA) ** 2 for k in range(3)]
        for a, b, n, k in rows:
            inside = []
            for c in range(10):
                idx = [0, 0, 0]
                idx[pa], idx[pb], idx[pc] = a, b, 9 - c if flip else c
                s = sq[0][idx[0]] + sq[1][idx[1]]
                if dim == 3:
                    s = s + sq[2][idx[2]]
                inside.append(bool(s < r * r))
            if n is None:  # all below the open sub-cell inside, all above outside
                opened += 1
                assert all(inside[:k]) and not any(inside[k + 1:]), (dim, r, xl, node, a, b)
            else:
                assert sum(inside) == n, (dim, r, xl, node, a, b, n)
    assert ruled > 10
    if rmax > 2.0:
        assert opened > 0  # the ties reach the exact decision
