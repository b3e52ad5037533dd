"""Factorizations whose bounded waits run out, at many limits, through the chain of small
blocks (clusters of 1, 8 and 16 CTAs, one and two leaves) and the diagonal tiles.

Whichever of a CTA's warps gives up first, and wherever the others are then, the stage
ends: with RGF_ETIMEOUT, or, where the limit was long enough, with the right factor.
The handle then factorizes with the default limit.  At one poll some wait always runs
out: a column is not there when the next one first looks.

Tolerance: test_gpu_panel.py's.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
RGF_ETIMEOUT = 5


@pytest.mark.parametrize("ns,nt,nd", [(10, 4, 1), (20, 4, 5), (32, 6, 0), (40, 6, 3), (64, 4, 8),
                                      (100, 2, 2), (160, 2, 0), (300, 2, 3)])
def test_stage_ends_at_every_limit(rgf, ns, nt, nd):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    logdet = O.logdet(layout, MF)
    tol = 8 * (ns + nd) * EPS * abs(logdet)
    with rgf.RGF(ia, ja, a, ns, nt, nd) as s:
        for polls in (1, 2, 3, 5, 8, 12, 16, 24, 32, 64, 128, 256, 1):
            s.set_wait_limit(polls)
            for _ in range(3):  # launched directly, then captured and replayed
                try:
                    s.factorize()
                    assert polls > 1
                    assert abs(s.logDet() - logdet) <= tol
                except rgf.RGFError as e:
                    assert e.status == RGF_ETIMEOUT
            s.set_wait_limit(0)
            s.factorize()
            assert abs(s.logDet() - logdet) <= tol
