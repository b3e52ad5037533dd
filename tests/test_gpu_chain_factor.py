"""The factorization of small blocks in one launch: block sizes around the 16-column
half, the leaf, the second leaf and the cluster sizes' lines, arrowheads up to the line
where the separate launches take over and past it, and enough block columns that every
buffer is used again; the column reported when a later block is not positive definite.

Tolerance: each entry of L is a sum of at most ns + nd products and the generator's
blocks have condition numbers below 10, so entries differ from the oracle's by at most
about 8 (ns + nd) eps of the largest one.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _factor_entries(ns, nt, nd, MF):
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


@pytest.mark.parametrize("nt", [1, 2, 6])
@pytest.mark.parametrize("ns,nd", [(1, 0), (1, 1), (1, 71), (3, 2), (8, 64), (11, 1), (12, 1), (16, 0),
                                   (17, 3), (24, 4), (24, 5), (30, 42), (30, 43), (31, 0), (32, 0),
                                   (33, 0), (33, 39), (42, 6), (48, 1), (63, 9), (64, 0), (64, 8),
                                   (64, 9), (65, 0)])
def test_factor(rgf, ns, nd, nt):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns * 7 + nd + nt)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    want = _factor_entries(ns, nt, nd, MF)
    with rgf.RGF(ia, ja, a, ns, nt, nd) as s:
        for _ in range(3):  # launched directly, then captured and replayed
            s.factorize()
            got = _factor_entries(ns, nt, nd, s.export_factor())
            assert np.max(np.abs(got - want)) <= 8 * (ns + nd) * EPS * np.max(np.abs(want))
        assert abs(s.logDet() - O.logdet(layout, MF)) <= 1e-12 * abs(O.logdet(layout, MF))


@pytest.mark.parametrize("ns,col", [(5, 2), (20, 17), (40, 3), (40, 37), (64, 63)])
def test_not_positive_definite_column(rgf, ns, col):
    nt, nd, bad = 4, 2, 2  # the pivot of column `col` of block 2 becomes negative
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns)
    a = a.copy()
    k = bad * ns + col
    a[int(ia[k])] = -1e3  # rows ascend within a column: the first entry is the diagonal one
    assert int(ja[int(ia[k])]) == k
    with rgf.RGF(ia, ja, a, ns, nt, nd) as s:
        with pytest.raises(rgf.RGFError):
            s.factorize()
        assert s.info()["not_spd_column"] == k
