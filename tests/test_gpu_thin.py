"""Thin FP64 products (the block substitution's n <= 16 and the arrowhead's
m <= 16): every column count of the dispatch and its neighbours, block sizes
around the kernels' 32-row tiles, 32-term K tiles and cluster split.

The solve's tolerance: the substitution is backward stable, so with the
well-conditioned generator matrices (condition number below 10) the error of
x stays within about 4 (ns + nd) eps of |x|_max.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("ns,nt,nd", [(5, 3, 2), (32, 2, 0), (33, 3, 1), (130, 3, 6), (257, 2, 16),
                                      (40, 3, 17)])
def test_solve_column_counts(rgf, ns, nt, nd):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    n = ns * nt + nd
    ref_layout = O.Layout(ns, nt, nd)
    MF = O.ingest(ref_layout, ia, ja, a)
    O.factorize(ref_layout, MF)
    tol = 4 * (ns + nd) * EPS
    with rgf.RGF(ia, ja, a, ns, nt, nd) as s:
        for nrhs in (1, 2, 3, 4, 5, 6, 7, 8, 11, 12, 13, 16, 17):
            b = gen.random_rhs(n, nrhs, nrhs)
            x = s.solve(np.empty((n, nrhs)), b, nrhs).reshape(n, nrhs)
            for q in (0, nrhs - 1):
                want = O.solve(ref_layout, MF, b[:, q].copy())
                assert np.max(np.abs(x[:, q] - want)) <= tol * np.max(np.abs(want)), (nrhs, q)


@pytest.mark.parametrize("ns,nt,nd", [(33, 3, 1), (64, 2, 3), (65, 3, 5), (100, 2, 9), (257, 3, 13),
                                      (45, 2, 16), (45, 2, 17)])
def test_arrowhead_row_counts(rgf, ns, nt, nd):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns * 3 + nd)
    ref = O.run_all(ns, nt, nd, ia, ja, a, exact=True)
    with rgf.RGF(ia, ja, a, ns, nt, nd) as s:
        assert abs(s.logDet() - ref["logdet"]) <= 1e-12 * abs(ref["logdet"])
        d = s.RGFdiag()
    assert np.max(np.abs(d - ref["diag"]) / np.abs(ref["diag"])) <= 4 * (ns + nd) * EPS
