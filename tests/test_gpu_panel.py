"""The panel factorization's kernels (diagonal tiles of up to 128 columns, rows
below them) against the oracle's factor: block sizes around the 16-column half,
the 32-column leaf and the 64- and 128-column tiles, row counts around each
rows-per-CTA rule, and the column reported for a matrix that is not SPD.

Tolerance: each entry of L is a sum of at most ns + nd products and the
generator's blocks have condition numbers below 10, so entries differ from the
oracle's by at most about 8 (ns + nd) eps of the largest one.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _lower(L, ns, nt, nd, MF):
    """The entries of MF that the factor defines (strict upper parts dropped)."""
    parts, pos = [], 0
    for i in range(nt):
        lda = (2 * ns if i < nt - 1 else ns) + nd
        P = MF[pos:pos + lda * ns].reshape(ns, lda)  # P[col, row]
        keep = np.arange(lda)[None, :] >= np.arange(ns)[:, None]
        parts.append(P[keep])
        pos += lda * ns
    if nd:
        parts.append(MF[pos:].reshape(nd, nd)[np.triu_indices(nd)])
    return np.concatenate(parts)


def _check(rgf, ns, nt, nd, precision="fp64", **knobs):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns * 7 + nd)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    with rgf.RGF(ia, ja, a, ns, nt, nd, precision=precision) as s:
        if knobs:
            s.set_tuning(**knobs)
        s.factorize()
        got = _lower(layout, ns, nt, nd, s.export_factor())
    want = _lower(layout, ns, nt, nd, MF)
    assert np.max(np.abs(got - want)) <= 8 * (ns + nd) * EPS * np.max(np.abs(want))


@pytest.mark.parametrize("ns", [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65, 95, 97, 127, 128,
                                129, 160, 193, 257])
@pytest.mark.parametrize("nd", [0, 5])
def test_tile_widths(rgf, ns, nd):
    _check(rgf, ns, 2, nd)


@pytest.mark.parametrize("ns,nt,nd", [(32, 1, 0), (40, 3, 130), (128, 1, 33), (620, 2, 3),
                                      (1290, 2, 1)])
def test_row_counts_and_corners(rgf, ns, nt, nd):
    _check(rgf, ns, nt, nd)


@pytest.mark.parametrize("knobs", [{"leaf_nb": 16}, {"leaf_nb": 64}, {"lookahead": 0},
                                   {"leaf_nb": 16, "lookahead": 0}])
def test_knobs(rgf, knobs):
    _check(rgf, 200, 2, 3, **knobs)


@pytest.mark.parametrize("col", [0, 1, 15, 16, 31, 32, 70, 127, 128, 149, 150, 290, 300])
def test_column_of_a_non_positive_pivot(rgf, col):
    ns, nt, nd = 150, 2, 3
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=9)
    a = a.copy()
    a[int(ia[col])] = -1.0  # the column's diagonal entry comes first
    with rgf.RGF(ia, ja, a, ns, nt, nd) as s:
        with pytest.raises(rgf.RGFError) as e:
            s.factorize()
        assert e.value.status == 3
        assert s.info()["not_spd_column"] == col


@pytest.mark.parametrize("ns", [130, 159, 161, 255, 287, 288, 289, 416, 417])
@pytest.mark.parametrize("nd", [0, 3, 150, 161])
def test_last_tiles_past_128(rgf, ns, nd):
    _check(rgf, ns, 2, nd)
