"""FP64 products whose K range a cluster splits, at the edges of the 32- and
64-wide tiles, of the 16-term K tiles and of the slices (slices without a term
among them), and the thin products next to them.

Error bound: a sum of K products in any order is within K eps |A| |B| of the exact
one, and so is the reference; plus the roundings of alpha, beta and the last sum.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("m,n", [(1, 1), (17, 17), (32, 32), (33, 31), (64, 65), (97, 128), (16, 130),
                                 (130, 16), (300, 333)])
@pytest.mark.parametrize("k", [1, 15, 16, 17, 127, 128, 129, 260, 1000])
@pytest.mark.parametrize("ta,tb", [("N", "T"), ("T", "N"), ("N", "N")])
def test_split_k(rgf, ta, tb, m, n, k):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    A = rng.standard_normal((k, m) if ta == "T" else (m, k))
    B = rng.standard_normal((n, k) if tb == "T" else (k, n))
    C0 = rng.standard_normal((m, n))
    dev = torch.device("cuda", 0)
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).to(dev)
    dB = torch.from_numpy(np.ascontiguousarray(B.T)).to(dev)
    opA = A.T if ta == "T" else A
    opB = B.T if tb == "T" else B
    for alpha, beta in ((-1.0, 1.0), (0.5, 0.0)):
        dC = torch.from_numpy(np.ascontiguousarray(C0.T)).to(dev)
        torch.cuda.synchronize()
        rgf.dgemm_device("fp64", ta, tb, m, n, k, alpha, dA.data_ptr(), A.shape[0], dB.data_ptr(),
                         B.shape[0], beta, dC.data_ptr(), m)
        ref = alpha * (opA @ opB) + beta * C0
        bound = 2 * (k + 2) * EPS * (np.abs(opA) @ np.abs(opB)) + 4 * EPS * np.abs(C0)
        assert np.all(np.abs(dC.cpu().numpy().T - ref) <= bound)
