"""Split products whose results leave FP64's normal range (the conversion's
rare path), in tiles of which only a part is written, with and without C.

Bound: 2e-11 of (|A||B|)_{rc} for the 40-bit operands, plus one subnormal unit
for the rounding of a result below the normal range.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(130, 70, 128), (5, 129, 320), (256, 256, 640)])
@pytest.mark.parametrize("scale", [1e-165, 1e-155, 1.0, 1e150])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)])
def test_result_range(rgf, m, n, k, scale, alpha, beta):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((m, k)) * scale
    B = rng.standard_normal((k, n)) * scale
    C0 = rng.standard_normal((m, n)) * scale * scale * 3.0
    dev = torch.device("cuda", 0)
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).to(dev)
    dB = torch.from_numpy(np.ascontiguousarray(B.T)).to(dev)
    dC = torch.from_numpy(np.ascontiguousarray(C0.T)).to(dev)
    torch.cuda.synchronize()
    rgf.dgemm_device("split", "N", "N", m, n, k, alpha, dA.data_ptr(), m, dB.data_ptr(), k, beta,
                     dC.data_ptr(), m)
    got = dC.cpu().numpy().T
    # the reference with the scale factored out, so that it does not lose bits itself
    As, Bs = A / scale, B / scale
    ref = (alpha * (As @ Bs)).astype(np.longdouble) * np.longdouble(scale) ** 2 + beta * C0.astype(
        np.longdouble)
    bound = np.abs(alpha) * (np.abs(As) @ np.abs(Bs)).astype(np.longdouble) * np.longdouble(scale) ** 2
    err = np.abs(got.astype(np.longdouble) - ref)
    assert np.all(np.isfinite(got))
    assert np.all(err <= 2e-11 * bound + 4e-16 * np.abs(ref) + 5e-324)
