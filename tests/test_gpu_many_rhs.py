"""Solves with more than 16 right-hand sides: block sizes and counts around the line between
the one-launch substitution and separate products, the column groups of those (8, 12, a
last one of 1) and the tiles past 512; wide arrowheads; FP64 and refined split solves.

Tolerance: test_gpu_solve_chain.py's.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("ns,nt,nd,counts", [
    (3, 4, 1, (17, 600)), (16, 4, 2, (255, 256, 257)), (64, 3, 0, (31, 32, 33)), (100, 3, 3, (17, 193, 204)),
    (144, 3, 2, (17, 24, 25)), (161, 2, 1, (17, 192, 193)), (257, 3, 4, (17, 64, 511, 512, 513)),
    (600, 2, 0, (18, 40, 200)), (33, 2, 90, (17, 65))])
def test_solve(rgf, precision, ns, nt, nd, counts):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    n = ns * nt + nd
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    tol = (4 if precision == "fp64" else 8) * (ns + nd) * EPS
    with rgf.RGF(ia, ja, a, ns, nt, nd, precision=precision) as s:
        for nrhs in counts:
            b = gen.random_rhs(n, nrhs, nrhs)
            want = np.stack([O.solve(layout, MF, b[:, q].copy()) for q in range(nrhs)], axis=1)
            for _ in range(3):  # launched directly, then captured and replayed
                x = np.asarray(s.solve(np.empty((n, nrhs), order="F"), b, nrhs)).reshape(n, nrhs)
                err = np.max(np.abs(x - want), axis=0) / np.max(np.abs(want), axis=0)
                assert np.max(err) <= tol, (nrhs, int(np.argmax(err)))
