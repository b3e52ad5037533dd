"""The selected inverse with arrowheads of more than one 64-column tile, in memory that an
earlier handle has used: the inverse of the corner is triangular and only its upper part
is written, so nothing may read the rest of the buffer.

The buffer comes back dirty through the device-memory cache: a solve whose right-hand
sides have as many entries as the diagonal blocks' inverses leaves its results in
buffers of just that size, one of which the next handle of the process is then given.

Tolerance (test_gpu_selinv_blocks.py): 16 (ns + nd) eps of the largest entry.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.fixture()
def dirty(rgf):
    """dirty(count): the next allocations of count doubles get used memory."""
    rgf.set_device_cache(1 << 30)

    def fill(count):
        nt, nd = divmod(count, 8)
        ia, ja, a = gen.generate_bta(8, nt, nd, seed=1)
        with rgf.RGF(ia, ja, a, 8, nt, nd) as s:
            b = 1.0 + np.abs(gen.random_rhs(count, 1, 5))
            x = s.solve(np.empty_like(b), b, 1)
            assert np.count_nonzero(x) == count
            s.RGFdiag()  # of that size, too
    yield fill
    rgf.set_device_cache(0)


@pytest.mark.parametrize("ns,nt,nd", [(10, 2, 63), (10, 2, 64), (10, 2, 65), (70, 3, 130), (100, 1, 129),
                                      (80, 2, 200)])
@pytest.mark.parametrize("selinv", ["exact", "compat"])
def test_selected_inverse_in_used_memory(rgf, dirty, ns, nt, nd, selinv):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    tol = 16 * (ns + nd) * EPS
    dirty(nt * ns * ns + nd * nd)
    with rgf.RGF(ia, ja, a, ns, nt, nd, selinv=selinv) as s:
        got = s.RGFdiag()
        want = (O.selinv_exact if selinv == "exact" else O.selinv_compat)(layout, MF)
        assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
        if selinv == "exact":
            _, want = O.selinv_exact(layout, MF, blocks=True)
            assert np.max(np.abs(s.export_selinv() - want)) <= tol * np.max(np.abs(want))


def test_hermitian_in_used_memory(rgf, dirty):
    """A complex arrowhead of 33 rows is one of 66 in the real embedding."""
    ns, nt, nd = 6, 3, 33
    rng = np.random.default_rng(4)
    n = ns * nt + nd
    H = np.zeros((n, n), dtype=np.complex128)
    for r in range(n):
        for c in range(r):
            if r >= ns * nt or r // ns - c // ns <= 1:
                H[r, c] = 0.3 * (rng.standard_normal() + 1j * rng.standard_normal())
    H = H + H.conj().T + np.diag(np.full(n, 2.0 * n))
    ia, ja, a = [0], [], []
    for c in range(n):
        rows = [r for r in range(c, n) if r == c or r >= ns * nt or r // ns - c // ns <= 1]
        ja += rows
        a += [H[r, c] for r in rows]
        ia.append(len(ja))
    dirty(nt * (2 * ns) ** 2 + (2 * nd) ** 2)
    with rgf.RGF(np.array(ia, dtype=np.uint64), np.array(ja, dtype=np.uint64), np.array(a), ns, nt,
                 nd) as s:
        want = np.diag(np.linalg.inv(H)).real
        # the embedding's blocks are twice as large
        assert np.max(np.abs(s.RGFdiag().real - want)) <= 32 * (ns + nd) * EPS * np.max(np.abs(want))


@pytest.mark.parametrize("precision,lookahead", [("fp64", 1), ("fp64", 0), ("split", 1)])
@pytest.mark.parametrize("ns,nt,nd", [(161, 1, 33), (161, 2, 40), (200, 5, 64), (300, 4, 100), (520, 3, 33)])
def test_corner_of_wide_arrowheads(rgf, precision, lookahead, ns, nt, nd, tmp_path, monkeypatch):
    """More rows than the one-pass corner update takes: with look-ahead the products of all
    block columns but the last run on its stream.  Tolerance: test_gpu_panel.py's; at 5
    slices test_gpu_selinv_blocks.py's."""
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=nd)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    want = np.triu(MF[-nd * nd:].reshape(nd, nd))
    tol = 8 * (ns + nd) * EPS + (4 * 2.0 ** (3 - 8 * 5) * (ns + nd) if precision == "split" else 0)
    path = tmp_path / "trace.csv"
    for traced in (False, True):
        if traced:
            monkeypatch.setenv("RGF_GB300_TRACE", str(path))
        with rgf.RGF(ia, ja, a, ns, nt, nd, precision=precision) as s:
            s.set_tuning(lookahead=lookahead, fp64_tile=32)
            for _ in range(1 if traced else 3):  # launched directly, then captured and replayed
                s.factorize()
                got = np.triu(s.export_factor()[-nd * nd:].reshape(nd, nd))
                assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
    rows = [ln.split(",") for ln in path.read_text().splitlines()]
    shape = f"fp64 cls0 m{nd} n{nd} k{ns} b1"
    streams = [r[2] for r in rows if r[3] == shape]
    assert streams == ["1" if lookahead else "0"] * (nt - 1) + ["0"]
