"""Factorizations of matrices far from 1 in magnitude, through the chain of small blocks,
the diagonal tiles (one to five leaves), the rows below them and the corner.

Scaling a matrix by 4^k scales its factor by 2^k and its inverse by 4^-k, exactly
in FP64 while nothing leaves the normal range; each scaled result is compared with the
oracle's for the unscaled matrix.  Tolerance: that of the unscaled matrix, 16 (ns + nd) eps of
the largest entry (test_gpu_panel.py, test_gpu_selinv_blocks.py); at 5 slices the
selected inverse's of test_gpu_selinv_blocks.py.

Pivots below the normal range: an entry of A and each A-sized intermediate carries an error
of up to 2^-1074, an entry of L is a sum of at most ns + nd of those over a diagonal
entry of at least sqrt(ns + 2) in units of the scale's root.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _entries(ns, nt, nd, MF):
    """The entries of MF that the factor defines (strict upper parts dropped)."""
    parts, pos = [], 0
    for i in range(nt):
        lda = (2 * ns if i < nt - 1 else ns) + nd
        P = MF[pos:pos + lda * ns].reshape(ns, lda)  # P[col, row]
        parts.append(P[np.arange(lda)[None, :] >= np.arange(ns)[:, None]])
        pos += lda * ns
    if nd:
        parts.append(MF[pos:].reshape(nd, nd)[np.triu_indices(nd)])
    return np.concatenate(parts)


SHAPES = [(2, 3, 1), (24, 3, 2), (40, 3, 3), (64, 2, 0), (100, 2, 1), (150, 2, 3), (300, 2, 2), (8, 3, 90)]


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("power", [-900, -600, -540, -520, 500, 514, 900])
@pytest.mark.parametrize("ns,nt,nd", SHAPES)
def test_scaled(rgf, precision, ns, nt, nd, power):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    want = _entries(ns, nt, nd, MF)
    diag = O.selinv_exact(layout, MF)
    n = ns * nt + nd
    logdet = O.logdet(layout, MF) + n * power * np.log(2.0)
    tol = 16 * (ns + nd) * EPS
    stol = tol + (4 * 2.0 ** (3 - 8 * 5) * (ns + nd) if precision == "split" else 0.0)
    with rgf.RGF(ia, ja, np.ldexp(a, power), ns, nt, nd, precision=precision) as s:
        s.factorize()
        got = np.ldexp(_entries(ns, nt, nd, s.export_factor()), -power // 2)
        assert np.max(np.abs(got - want)) <= stol * np.max(np.abs(want))
        assert abs(s.logDet() - logdet) <= 1e-12 * abs(logdet)
        got = np.ldexp(s.RGFdiag(), power)
        assert np.max(np.abs(got - diag)) <= stol * np.max(np.abs(diag))


@pytest.mark.parametrize("power", [-1040, -1028])
@pytest.mark.parametrize("ns,nt,nd", SHAPES)
def test_subnormal_pivots(rgf, ns, nt, nd, power):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    a = np.ldexp(np.ldexp(a, power), -power)  # as the scaled matrix holds them
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    want = _entries(ns, nt, nd, MF)
    unit = 2.0 ** (-1074 - power)  # the spacing of A-sized values, scaled back
    tol = 16 * (ns + nd) * EPS * np.max(np.abs(want)) + (ns + nd) * unit / np.sqrt(ns + 2.0)
    with rgf.RGF(ia, ja, np.ldexp(a, power), ns, nt, nd) as s:
        s.factorize()
        got = np.ldexp(_entries(ns, nt, nd, s.export_factor()), -power // 2)
        assert np.max(np.abs(got - want)) <= tol


def test_pivot_reciprocals(rgf):
    """Second pivots of 2 x 2 blocks, c - v^2 / d, over mantissas and exponents of d (v^2 / d
    as large as c / 2): the reciprocal and the product in front of it are within a few
    units, so L_22 = sqrt(c - v^2 / d) is within 4 eps."""
    nt = 20000
    rng = np.random.default_rng(11)
    e = rng.integers(-1020, 1016, nt)
    d = np.ldexp(1.0 + rng.random(nt), e)
    # c between 2^-1000 and 2^1000, v = sqrt(d c / 2): its exponent is the mean of theirs
    f = rng.integers(-1000, 1000, nt)
    c = np.ldexp(1.0 + rng.random(nt), f)
    l = np.sqrt(0.5) * np.sqrt(c)       # L_21 = v / sqrt(d)
    v = l * np.sqrt(d)
    ia = np.concatenate([[0], np.cumsum(np.tile([2, 1], nt))]).astype(np.uint64)
    ja = np.stack([2 * np.arange(nt), 2 * np.arange(nt) + 1, 2 * np.arange(nt) + 1], 1).ravel().astype(np.uint64)
    a = np.stack([d, v, c], 1).ravel()
    with rgf.RGF(ia, ja, a, 2, nt, 0) as s:
        s.factorize()
        MF = s.export_factor()
    P = np.concatenate([MF[:-4].reshape(nt - 1, 2, 4)[:, :, :2], MF[-4:].reshape(1, 2, 2)])  # [block, col, row]
    ld, lc, lv = (x.astype(np.longdouble) for x in (d, c, v))
    want11, want21 = np.sqrt(ld), lv / np.sqrt(ld)
    want22 = np.sqrt(lc - lv * (lv / ld))
    for got, want, k in ((P[:, 0, 0], want11, 2), (P[:, 0, 1], want21, 3), (P[:, 1, 1], want22, 4)):
        assert np.max(np.abs(got.astype(np.longdouble) / want - 1)) <= k * EPS


@pytest.mark.parametrize("ns,nt,nd", SHAPES)
def test_graded(rgf, ns, nt, nd):
    """Rows and columns scaled by powers of two between 2^-220 and 2^220 each, so that magnitudes
    from 2^-440 to 2^440 stand side by side: the factor's rows scale alike, exactly."""
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    n = ns * nt + nd
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    want = _entries(ns, nt, nd, MF)
    diag = O.selinv_exact(layout, MF)
    e = 2 * np.random.default_rng(ns).integers(-110, 111, n)
    row, col = ja.astype(np.int64), np.repeat(np.arange(n), np.diff(ia.astype(np.int64)))
    rows = []  # the row of each entry of _entries
    for i in range(nt):
        r = np.arange(i * ns, min(i + 2, nt) * ns)
        r = np.concatenate([r, np.arange(nt * ns, n)])
        rows += [r[c:] for c in range(ns)]
    rows += [np.arange(nt * ns + c, n) for c in range(nd)]
    tol = 16 * (ns + nd) * EPS
    with rgf.RGF(ia, ja, np.ldexp(a, e[row] + e[col]), ns, nt, nd) as s:
        s.factorize()
        got = np.ldexp(_entries(ns, nt, nd, s.export_factor()), -e[np.concatenate(rows)])
        assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
        got = np.ldexp(s.RGFdiag(), 2 * e)
        assert np.max(np.abs(got - diag)) <= tol * np.max(np.abs(diag))
