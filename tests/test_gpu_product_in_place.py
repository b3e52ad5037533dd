"""The split engine's in-place product X := X U, and the FP64 product that stands in for it
when the operands cannot be described to the tensor cores' copies: one to many tiles, all
of whose CTAs read rows that others write.

Tolerance: sums of at most k terms, in FP64 or with 55-bit operands: 2 k eps of
(|X| |U|) and of the largest entries' product.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("maps", [True, False])
@pytest.mark.parametrize("m,k", [(1, 64), (5, 65), (129, 100), (300, 384), (1472, 256), (2006, 512)])
def test_product(rgf, m, k, maps):
    rng = np.random.default_rng(m + k)
    X = rng.standard_normal((m, k))
    U = np.triu(rng.standard_normal((k, k))) + np.tril(np.full((k, k), np.nan), -1)
    Uz = np.triu(np.nan_to_num(U))
    for _ in range(3):
        got = rgf.debug_product_in_place(X, U, maps)
        assert np.all(np.abs(got - X @ Uz) <= 2 * k * EPS * (np.abs(X) @ np.abs(Uz) +
                                                         np.abs(X).max() * np.abs(Uz).max()))
