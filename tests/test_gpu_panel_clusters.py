"""The diagonal tile by itself, by clusters of 16 thread blocks and by the 8 that a device
without room for 16 gets: widths around the leaf, the rows of a worker and the widest tile,
and a pivot that is not positive.

Tolerance: test_gpu_panel.py's, 8 w eps of the largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _tile(w):
    A = np.random.default_rng(w).standard_normal((w, w))
    return A @ A.T / w + (w + 2.0) * np.eye(w)


@pytest.mark.parametrize("ctas", [8, 16])
@pytest.mark.parametrize("w", [1, 31, 32, 33, 39, 47, 64, 65, 96, 127, 128, 129, 137, 143, 144, 145, 146,
                               152, 159, 160])
def test_tile(rgf, w, ctas):
    A = _tile(w)
    want = np.linalg.cholesky(A)
    got = rgf.debug_panel_tile(A, ctas)
    assert np.max(np.abs(got - want)) <= 8 * w * EPS * np.max(np.abs(want))


@pytest.mark.parametrize("ctas", [8, 16])
def test_not_positive_definite(rgf, ctas):
    A = _tile(160)
    A[150, 150] = -1.0
    with pytest.raises(rgf.RGFError) as e:
        rgf.debug_panel_tile(A, ctas)
    assert e.value.status == 3
    for w, c in ((0, 8), (161, 8), (32, 4)):
        with pytest.raises(rgf.RGFError) as e:
            rgf.debug_panel_tile(np.eye(w), c)
        assert e.value.status == 1
