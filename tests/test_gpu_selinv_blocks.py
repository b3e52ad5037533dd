"""All blocks of the selected inverse (Sigma_ii, Sigma_{i+1,i}, Sigma_{d,i}, Sigma_dd)
against the oracle's: block sizes around the 32-wide tiles of the symmetric copy
and the 16- and 32-column rules, arrowheads of 0, 1, 32 and more rows, one to many block
columns (in more than one batch of K_i), and split precision on both sides of the
line between FP64 and sliced products.

Tolerance: the generator's blocks have condition numbers below 10 and an entry of
Sigma is a chain of sums of at most ns + nd terms over the block columns that the
recursion damps, so FP64 entries differ by at most about 16 (ns + nd) eps of the
largest one.  At S slices an operand keeps 8 S - 1 bits of its row's largest magnitude:
each of the four products of a block adds at most 2^(3 - 8 S) (ns + nd) of the largest
entries' product.
"""
import numpy as np
import pytest

from oracle import rgf_oracle as O
from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _check(rgf, ns, nt, nd, precision="fp64", repeat=1):
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns * 5 + nt + nd)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    _, want = O.selinv_exact(layout, MF, blocks=True)
    tol = 16 * (ns + nd) * EPS
    if precision == "split":
        tol += 4 * 2.0 ** (3 - 8 * 5) * (ns + nd)
    with rgf.RGF(ia, ja, a, ns, nt, nd, precision=precision) as s:
        for _ in range(repeat):  # launched directly, then captured and replayed
            s.factorize()
            got = s.export_selinv()
            assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))


@pytest.mark.parametrize("ns", [1, 2, 5, 11, 12, 13, 16, 17, 28, 29, 31, 32, 33, 42, 48, 56, 63, 64, 65, 72, 73,
                                100, 129])
@pytest.mark.parametrize("nt,nd", [(1, 0), (2, 1), (5, 0), (4, 6), (3, 17), (3, 33)])
def test_blocks(rgf, ns, nt, nd):
    _check(rgf, ns, nt, nd, repeat=3)


@pytest.mark.parametrize("ns,nd", [(100, 2), (230, 6), (260, 0), (300, 5), (300, 0), (520, 20)])
def test_split_lines(rgf, ns, nd):
    _check(rgf, ns, 4, nd, "split", repeat=3)


def test_batches_of_k(rgf):
    _check(rgf, 1500, 10, 3)


@pytest.mark.parametrize("ns,nt,nd", [(1450, 2, 0), (1460, 3, 2), (1664, 2, 6)])
def test_column_groups(rgf, ns, nt, nd):
    """Blocks large enough that the rows below them are solved by group inverses: the
    factor's entries too (bulk products at 5 slices, as above)."""
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=ns + nd)
    layout = O.Layout(ns, nt, nd)
    MF = O.ingest(layout, ia, ja, a)
    O.factorize(layout, MF)
    _, want = O.selinv_exact(layout, MF, blocks=True)
    tol = 16 * (ns + nd) * EPS + 4 * 2.0 ** (3 - 8 * 5) * (ns + nd)
    with rgf.RGF(ia, ja, a, ns, nt, nd, precision="split") as s:
        for _ in range(3):
            s.factorize()
            got = s.export_factor()
            pos = 0
            for i in range(nt):
                lda = (2 * ns if i < nt - 1 else ns) + nd
                keep = np.arange(lda)[None, :] >= np.arange(ns)[:, None]
                g = got[pos:pos + lda * ns].reshape(ns, lda)[keep]
                w = MF[pos:pos + lda * ns].reshape(ns, lda)[keep]
                assert np.max(np.abs(g - w)) <= tol * np.max(np.abs(w))
                pos += lda * ns
            sig = s.export_selinv()
            assert np.max(np.abs(sig - want)) <= tol * np.max(np.abs(want))
