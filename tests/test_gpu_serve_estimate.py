"""The memory that the server reserves for a factorization covers what its handle takes, in
the factorization and the selected inversion: long chains with arrowheads up to the widest
of the one-pass corner update, both precisions, both recursions.  The factors stay
right where block columns share a partial sum of that update."""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("ns,nt,nd,opts", [(3, 20000, 32, {}), (3, 20000, 32, {"precision": "split"}),
                                           (40, 1500, 31, {}), (300, 30, 32, {"precision": "split"}),
                                           (20, 400, 6, {"selinv": "compat"}), (600, 4, 33, {})])
def test_reservation_covers_the_handle(rgf, ns, nt, nd, opts):
    m = gen.generate_bta(ns, nt, nd, seed=12)
    srv = rgf.RGFServer(hbm_budget_bytes=4 << 30, slots=1, **opts)
    f = srv.wait(srv.submit_factor(*m, ns, nt, nd))
    assert f["status"] == 0
    st = srv.stats()
    assert st["arena_in_use"] <= st["used_bytes"]
    assert srv.wait(srv.submit_diag(f["factor_id"], ns * nt + nd))["status"] == 0
    st = srv.stats()
    assert st["arena_in_use"] <= st["used_bytes"] and st["arena_fallbacks"] == 0
    srv.close()


@pytest.mark.parametrize("ns,nt,nd", [(2, 1216, 3), (2, 1217, 32), (5, 2500, 2), (300, 609, 1)])
def test_corner_over_many_block_columns(rgf, ns, nt, nd):
    """Entries of the corner are sums of ns nt products over at most sqrt(nt + 2)."""
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=13)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    want = np.triu(MF[-nd * nd:].reshape(nd, nd))
    with rgf.RGF(ia, ja, a, ns, nt, nd) as s:
        s.factorize()
        got = np.triu(s.export_factor()[-nd * nd:].reshape(nd, nd))
    assert np.max(np.abs(got - want)) <= 2 * np.sqrt(ns * nt) * EPS * nd * np.max(np.abs(want))
