"""Residual block and norms of wide blocks: few rows to a chunk, one column block more than the
rows need, and the bounds of the workspace for narrower blocks and fewer rows. Reference and
bounds as in test_residual_norms_gpu.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,m", [(1, 2048), (9, 4100), (50, 2048), (1000, 700), (301, 1402),
                                 (77, 1025), (1200, 2048), (5000, 129)])
def test_wide_blocks(n, m, dtype):
    from fasteig_b200 import ops
    g = torch.Generator().manual_seed(n + m)
    AX, X, R = (torch.randn(n, m, generator=g, dtype=torch.float64).to(dtype).cuda()
                for _ in range(3))
    lam = torch.randn(m, generator=g, dtype=torch.float64).cuda()
    rn, xn, rel = ops.residual_norms(AX, X, lam, None, R)
    a, x, l = AX.double().cpu().numpy(), X.double().cpu().numpy(), lam.cpu().numpy()
    got = R.double().cpu().numpy()
    eps = torch.finfo(dtype).eps
    assert np.all(np.abs(got - (a - l * x)) <= (eps + 4e-16) * (np.abs(a) + np.abs(l * x)))
    tol = (n + 8) * 2.3e-16
    np.testing.assert_allclose(rn.cpu().numpy(), np.linalg.norm(got, axis=0), rtol=tol)
    np.testing.assert_allclose(xn.cpu().numpy(), np.linalg.norm(x, axis=0), rtol=tol)
    np.testing.assert_allclose(rel.cpu().numpy(),
                               np.linalg.norm(got, axis=0) / ((1 + np.abs(l)) * np.linalg.norm(x, axis=0)),
                               rtol=2 * tol)
    np.testing.assert_allclose(ops.column_norms(X).cpu().numpy(), np.linalg.norm(x, axis=0),
                               rtol=tol)


@pytest.mark.parametrize("n,m", [(1, 1), (63, 45), (1000, 700), (5000, 129), (20000, 2048)])
def test_workspace_bounds_smaller_calls(n, m):
    """A workspace for n x m serves every smaller block (a solver allocates it once)."""
    import fasteig_b200 as fe
    need = fe.lib.fe_residual_workspace_bytes(n, m)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    X = torch.randn(n, m, dtype=torch.float64, device="cuda")
    out = torch.empty(m, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for k in sorted({1, m // 3 + 1, m // 2 + 1, m - m // 7, m}):
        for r in sorted({1, n // 2 + 1, n}):
            if k <= m:
                assert fe.lib.fe_column_norms_f64(X.data_ptr(), m, r, k, out.data_ptr(),
                                                  ws.data_ptr(), need, s) == 0
