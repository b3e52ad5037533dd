"""A caller's slice count above the default holds for the whole factorization and the
selected inverse: what is not a product at that count is FP64, entry by entry.

The matrices let every product with a small result be exact, so that FP64's relative
error of an entry stays a few units however small the entry is beside its row's largest
one, where operands cut at a fixed number of bits below a row's largest entry lose it.
"""
import numpy as np
import pytest

from rgf_gb300 import gen

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("slices", [6, 7, 8])
def test_rows_below_large_blocks(rgf, slices):
    """Diagonal D_0: L_10 = B D_0^{-1/2}, one product per entry (the square root, its
    reciprocal and the product: at most 4 eps), with columns of B down to 1e-14."""
    ns, nt, nd = 1460, 2, 2
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=6)
    col = np.repeat(np.arange(ns * nt + nd), np.diff(ia.astype(np.int64)))
    row = ja.astype(np.int64)
    a = a.copy()
    first = col < ns
    a[first & (row < ns) & (row != col)] = 0.0
    below = first & (row >= ns)
    a[below] *= 10.0 ** -(col[below] % 15)
    with rgf.RGF(ia, ja, a, ns, nt, nd, precision="split", slices=slices) as s:
        s.factorize()
        got = s.export_factor()[:ns * (2 * ns + nd)].reshape(ns, 2 * ns + nd)[:, ns:]
    diag = a[first & (row == col)]
    want = a[below].reshape(ns, ns + nd) / np.sqrt(diag)[:, None]
    assert np.max(np.abs(got / want - 1.0)) <= 4 * EPS


def _dense(D):
    n = D.shape[0]
    ia = np.concatenate([[0], np.cumsum(n - np.arange(n))]).astype(np.uint64)
    ja = np.concatenate([np.arange(c, n) for c in range(n)]).astype(np.uint64)
    return ia, ja, np.concatenate([D[c:, c] for c in range(n)])


@pytest.mark.parametrize("slices", [6, 7, 8])
def test_inverse_below_the_slicing_line(rgf, slices):
    """D = I + e S with |S_rc| in [1, 2): D^{-1} = I - e S + e^2 S^2 up to e^2 ns of its small
    entries.  Each of them is one entry of L, turned and carried through U U^T by products
    with 1: at most 32 eps with the reference's own."""
    ns, e = 256, 1e-9
    rng = np.random.default_rng(8)
    S = np.triu(rng.choice([-1.0, 1.0], (ns, ns)) * (1.0 + rng.random((ns, ns))), 1)
    S = S + S.T
    ia, ja, a = _dense(np.eye(ns) + e * S)
    with rgf.RGF(ia, ja, a, ns, 1, 0, precision="split", slices=slices) as s:
        got = s.export_selinv().reshape(ns, ns)
    off = ~np.eye(ns, dtype=bool)
    want = (-e * S + e * e * (S @ S))[off]
    assert np.max(np.abs(got[off] / want - 1.0)) <= 32 * EPS


@pytest.mark.parametrize("slices", [6, 7, 8])
def test_update_below_the_slicing_line(rgf, slices):
    """D_0 = 4 I, so L_10 = B / 2.  The odd rows of B hold 1 in column 0 and 1e-9 elsewhere, the
    even ones 0 and 1: an entry of L_11 in an odd row and an even column (or the other
    way round) is a sum of at most ns products of about 1e-9, off by 8 ns eps of the largest."""
    ns, nt, nd = 256, 3, 3
    ia, ja, a = gen.generate_bta(ns, nt, nd, seed=7)
    col = np.repeat(np.arange(ns * nt + nd), np.diff(ia.astype(np.int64)))
    row = ja.astype(np.int64)
    a = np.zeros_like(a)
    a[row == col] = 4.0
    second = (col >= ns) & (col < 2 * ns) & (row == col)
    a[second] = 2e4  # B B^T / 4 reaches 4.7e3
    below = (col < ns) & (row >= ns) & (row < 2 * ns)
    B = np.random.default_rng(9).uniform(0.5, 1.0, (ns, ns))
    odd = np.arange(ns) % 2 == 1
    B[odd, 0], B[~odd, 0] = 1.0, 0.0
    B[odd, 1:] *= 1e-9
    a[below] = B.T.reshape(-1)
    with rgf.RGF(ia, ja, a, ns, nt, nd, precision="split", slices=slices) as s:
        s.factorize()
        P = ns * (2 * ns + nd)
        got = np.tril(s.export_factor()[P:2 * P].reshape(ns, 2 * ns + nd)[:, :ns].T)
    F = (B / 2.0).astype(np.longdouble)
    A = 2e4 * np.eye(ns, dtype=np.longdouble) - F @ F.T
    want = np.zeros_like(A)
    for j in range(ns):
        want[j, j] = np.sqrt(A[j, j])
        want[j + 1:, j] = A[j + 1:, j] / want[j, j]
        A[j + 1:, j + 1:] -= np.outer(want[j + 1:, j], want[j + 1:, j])
    small = np.tril(odd[:, None] != odd[None, :])
    assert np.max(np.abs(got - want)[small]) <= 8 * ns * EPS * np.max(np.abs(want[small]))
