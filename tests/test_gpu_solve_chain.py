"""Block substitution in one launch and its lines: block sizes around the cluster sizes'
lines and the last ones it takes (144; 176 with one right-hand side), no and wide
arrowheads, one block, one to many right-hand sides (more than fit its shared memory,
too), FP64 and refined split solves.

Tolerance: the substitution is backward stable, so with the well-conditioned
generator matrices (condition number below 10) the error of x stays within about
4 (ns + nd) eps of |x|_max; the refined split solve stops at residuals of that size.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("ns,nt,nd", [(1, 1, 0), (1, 5, 1), (7, 1, 3), (3, 40, 2), (20, 4, 0), (20, 3, 60),
                                      (46, 3, 2), (47, 3, 2), (64, 3, 0), (100, 2, 1), (144, 3, 3), (145, 3, 3), (175, 3, 3),
                                      (176, 3, 1), (177, 3, 1), (256, 3, 4), (257, 3, 0), (250, 2, 80)])
def test_solve(rgf, precision, ns, nt, nd):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    n = ns * nt + nd
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    tol = (4 if precision == "fp64" else 8) * (ns + nd) * EPS
    with rgf.RGF(ia, ja, a, ns, nt, nd, precision=precision) as s:
        for nrhs in (1, 1, 1, 2, 5, 16, 100):
            b = gen.random_rhs(n, nrhs, nrhs)
            x = np.asarray(s.solve(np.empty((n, nrhs), order="F"), b, nrhs)).reshape(n, nrhs)
            for q in (0, nrhs // 2, nrhs - 1):
                want = O.solve(layout, MF, b[:, q].copy())
                assert np.max(np.abs(x[:, q] - want)) <= tol * np.max(np.abs(want)), (nrhs, q)
