"""With the look-ahead knob at 0 every stage stays on the handle's one stream, with the
results of the default within the usual bounds (test_gpu_selinv_blocks.py); with it the
selected inversion uses the second one, too."""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("ns,nt,nd", [(200, 3, 2), (300, 4, 5), (330, 3, 70)])
def test_streams(rgf, precision, ns, nt, nd, tmp_path, monkeypatch):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=3)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    want = O.selinv_exact(layout, MF)
    tol = 16 * (ns + nd) * EPS + (4 * 2.0 ** (3 - 8 * 5) * (ns + nd) if precision == "split" else 0)
    for lookahead in (0, 1):
        path = tmp_path / f"trace{lookahead}.csv"
        monkeypatch.setenv("RGF_GB300_TRACE", str(path))
        with rgf.RGF(ia, ja, a, ns, nt, nd, precision=precision) as s:
            s.set_tuning(lookahead=lookahead, fp64_tile=32)
            assert np.max(np.abs(s.RGFdiag() - want)) <= tol * np.max(np.abs(want))
        rows = [ln.split(",") for ln in path.read_text().splitlines()]
        assert {r[2] for r in rows} == ({"0", "1"} if lookahead else {"0"})
        monkeypatch.delenv("RGF_GB300_TRACE")
        with rgf.RGF(ia, ja, a, ns, nt, nd, precision=precision) as s:
            s.set_tuning(lookahead=lookahead, fp64_tile=32)
            for _ in range(3):  # launched directly, then captured and replayed
                s.factorize()
                assert np.max(np.abs(s.RGFdiag() - want)) <= tol * np.max(np.abs(want))
