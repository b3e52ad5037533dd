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
