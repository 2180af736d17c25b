"""Residual block and column norms at the edges of the kernel's row shares and column
blocks: one row, fewer rows than shares, more columns than a CTA takes, odd columns and
pitches (element-wide lanes), with and without B and R. Reference: NumPy in 64 bits. Norms
are sums of n squares in FP64: n eps of the sum; R is one rounding of the type past the FP64
product and difference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,m,ld", [(1, 1, 1), (3, 8, 8), (63, 45, 48), (129, 45, 45),
                                    (1000, 96, 96), (2311, 12, 16), (777, 1026, 1028),
                                    (300, 2052, 2052), (150, 515, 515)])
@pytest.mark.parametrize("with_b", [False, True])
def test_residual_norms(n, m, ld, dtype, with_b):
    from fasteig_b200 import ops
    g = torch.Generator().manual_seed(n + m)

    def block():
        t = torch.randn(n, ld, generator=g, dtype=torch.float64).to(dtype).cuda()
        return t[:, :m]

    AX, X, R = block(), block(), block()
    BX = block() if with_b else None
    lam = torch.randn(m, generator=g, dtype=torch.float64).cuda()
    rn, xn, rel = ops.residual_norms(AX, X, lam, BX, R)
    a = AX.double().cpu().numpy()
    x = (BX if with_b else X).double().cpu().numpy()
    l = lam.cpu().numpy()
    ref = a - l * x
    eps = torch.finfo(dtype).eps
    got = R.double().cpu().numpy()
    assert np.all(np.abs(got - ref) <= (eps + 4e-16) * (np.abs(a) + np.abs(l * x)))
    tol = (n + 8) * 2.3e-16
    np.testing.assert_allclose(rn.cpu().numpy(), np.linalg.norm(got, axis=0), rtol=tol)
    np.testing.assert_allclose(xn.cpu().numpy(), np.linalg.norm(x, axis=0), rtol=tol)
    np.testing.assert_allclose(rel.cpu().numpy(),
                               np.linalg.norm(got, axis=0) / ((1 + np.abs(l)) * np.linalg.norm(x, axis=0)),
                               rtol=2 * tol)
    np.testing.assert_allclose(ops.column_norms(X).cpu().numpy(),
                               np.linalg.norm(X.double().cpu().numpy(), axis=0), rtol=tol)
