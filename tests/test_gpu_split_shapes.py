"""Split products at the edges of the slicing and split-K rules: K around the
64-term atom, the 128- and 256-term parts of a slicing cluster and the longest K
it takes (2048), row counts around the 32-row blocks and 128-row tiles, operand
orientations, and digit counts with and without their own code.

Error bound, with M = max|A_r| max|B_c|: an S-digit operand keeps 8 S - 1 bits of
its row's largest magnitude, so the cut operands contribute at most
2^(3 - 8 S) K M; the 64-bit fixed-point sum drops cs = max(0, ceil(log2(1.03 K) +
8 (S + 1) - 2) - 62) bits with a rounding of half a unit, 2^(cs - 8 (S + 1) + 2) times
at most 4 M, in each of at most S (S + 1) / 2 ceil(K / 64) partial sums; then FP64
rounding of the result and of the reference.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _check(rgf, ta, tb, m, n, k, slices, alpha=-1.0, beta=1.0):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(m * 7 + n * 3 + k + slices)
    A = rng.standard_normal((k, m) if ta == "T" else (m, k))
    B = rng.standard_normal((n, k) if tb == "T" else (k, n))
    A[A.shape[0] // 2] *= 1e-9  # rows (columns) of different magnitude
    B[:, B.shape[1] // 3] *= 1e7
    C0 = rng.standard_normal((m, n))
    dev = torch.device("cuda", 0)
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).to(dev)
    dB = torch.from_numpy(np.ascontiguousarray(B.T)).to(dev)
    dC = torch.from_numpy(np.ascontiguousarray(C0.T)).to(dev)
    torch.cuda.synchronize()
    rgf.dgemm_device("split", ta, tb, m, n, k, alpha, dA.data_ptr(), A.shape[0], dB.data_ptr(),
                     B.shape[0], beta, dC.data_ptr(), m, slices=slices)
    got = dC.cpu().numpy().T
    opA = A.T if ta == "T" else A
    opB = B.T if tb == "T" else B
    ref = alpha * (opA @ opB) + beta * C0
    cs = max(0, int(np.ceil(np.log2(1.03 * k) + 8 * (slices + 1) - 2)) - 62)
    sums = slices * (slices + 1) // 2 * -(-k // 64)
    unit = 2.0 ** (3 - 8 * slices) * k
    if cs:
        unit += 0.5 * sums * 4 * 2.0 ** (cs - 8 * (slices + 1) + 2)
    bound = unit * np.abs(opA).max(1)[:, None] * np.abs(opB).max(0)[None, :]
    fp64 = 2 * k * EPS * (np.abs(opA) @ np.abs(opB)) + 4 * EPS * np.abs(C0)
    assert np.all(np.abs(got - ref) <= bound + fp64)


@pytest.mark.parametrize("k", [64, 65, 127, 128, 129, 192, 511, 513, 576, 1024, 1025, 2047, 2048, 2049])
@pytest.mark.parametrize("ta,tb", [("N", "T"), ("T", "N")])
def test_terms(rgf, ta, tb, k):
    _check(rgf, ta, tb, 130, 97, k, 5)


@pytest.mark.parametrize("m,n", [(1, 1), (31, 33), (128, 128), (129, 257), (700, 40), (1200, 300)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
def test_tiles(rgf, ta, tb, m, n):
    _check(rgf, ta, tb, m, n, 384, 7)


@pytest.mark.parametrize("slices", [1, 2, 3, 4, 5, 6, 7, 8])
def test_digits(rgf, slices):
    _check(rgf, "N", "T", 200, 150, 320, slices)
    _check(rgf, "T", "N", 200, 150, 1100, slices, alpha=1.0, beta=0.0)
