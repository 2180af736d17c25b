"""Cholesky and triangular inverse at the edges of their 32-wide blocks, of the staged
panel (512 rows) and of the largest inverse in shared memory (608), with a leading dimension
past k, and a failing pivot in the first, an inner and the last block. Bounds: the backward
errors of the factorization and of the inverse, c k eps, with c = 8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _spd(k, seed):
    g = torch.Generator().manual_seed(seed)
    M = torch.randn(2 * k + 3, k, generator=g, dtype=torch.float64)
    return (M.T @ M / (2 * k + 3)).numpy()


@pytest.mark.parametrize("k,ld", [(1, 1), (7, 9), (31, 31), (32, 32), (33, 40), (64, 64),
                                  (95, 97), (257, 257), (320, 320), (545, 545), (608, 608),
                                  (611, 611)])
def test_factor_and_inverse(k, ld):
    import fasteig_b200 as fe
    G = _spd(k, k)
    buf = np.full((k, ld), np.nan)  # column-major k x k with leading dimension ld
    buf[:, :k] = G
    dG = torch.from_numpy(buf).cuda()
    dI = torch.full((k, ld), float("nan"), dtype=torch.float64, device="cuda")
    info = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert fe.lib.fe_potrf_upper_f64(dG.data_ptr(), k, ld, info.data_ptr(), s) == 0
    assert fe.lib.fe_trinv_upper_f64(dG.data_ptr(), ld, dI.data_ptr(), ld, k, s) == 0
    R = dG.cpu().numpy()[:, :k].T
    X = dI.cpu().numpy()[:, :k].T
    assert info.item() == 0
    assert np.array_equal(R, np.triu(R)) and np.array_equal(X, np.triu(X))
    eps = 2.2e-16
    assert np.abs(R.T @ R - G).max() <= 8 * k * eps * np.abs(G).max()
    assert np.abs(X @ R - np.eye(k)).max() <= 8 * k * eps * (np.abs(X) @ np.abs(R)).max()


@pytest.mark.parametrize("k,pivot", [(5, 0), (64, 31), (64, 32), (100, 99), (300, 150)])
@pytest.mark.parametrize("value", [-1.0, 0.0, float("nan"), float("inf")])
def test_failing_pivot(k, pivot, value):
    from fasteig_b200 import ops
    G = np.diag(np.arange(1.0, k + 1))
    G[pivot, pivot] = value
    _, info = ops.potrf_upper(torch.from_numpy(G).cuda())
    assert info.item() == pivot + 1
