"""The one-CTA tridiagonalization (sizes up to 128, 256 or 512 threads) and the eigenvectors'
solves at the edges of its lane slots, of its thread counts and of its range, against NumPy:
random, clustered and already tridiagonal matrices. Bounds as in test_syevd_gpu.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("k", [1, 2, 3, 31, 32, 33, 48, 49, 64, 65, 97, 128, 129])
@pytest.mark.parametrize("kind", ["random", "near_identity", "tridiagonal"])
def test_small_eigenproblems(k, kind):
    import fasteig_b200 as fe
    rng = np.random.default_rng(k)
    M = rng.standard_normal((k, k))
    if kind == "random":
        A = M + M.T
    elif kind == "near_identity":
        A = np.eye(k) + 1e-9 * (M + M.T)
    else:
        A = 2 * np.eye(k) - np.eye(k, k=1) - np.eye(k, k=-1)
    dA = torch.from_numpy(A.copy()).cuda()
    W = torch.zeros(k, dtype=torch.float64, device="cuda")
    info = torch.ones(1, dtype=torch.int32, device="cuda")
    need = fe.lib.fe_syevd_f64_workspace_bytes(k)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert fe.lib.fe_syevd_f64(dA.data_ptr(), k, k, W.data_ptr(), info.data_ptr(), ws.data_ptr(),
                               need, torch.cuda.current_stream().cuda_stream) == 0
    assert info.item() == 0
    w, Z = W.cpu().numpy(), dA.cpu().numpy().reshape(k, k).T
    nrm = np.abs(A).sum(axis=1).max()
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-12 * nrm
    assert np.abs(A @ Z - Z * w[None, :]).max() <= 1e-12 * nrm
    assert np.abs(Z.T @ Z - np.eye(k)).max() <= 1e-12 * max(k, 10) / 10


@pytest.mark.parametrize("k", [12, 127, 160, 384, 385])
@pytest.mark.parametrize("length", [1, 2, 3, 4, 5, 9])
def test_eigenvector_clusters(k, length):
    """Clusters of one to nine equal eigenvalues (to 1e-9 of the norm), which start at every
    position of a CTA's four warps: vectors shared among the warps or done by one."""
    import fasteig_b200 as fe
    rng = np.random.default_rng(100 * k + length)
    Q = np.linalg.qr(rng.standard_normal((k, k)))[0]
    lam = np.repeat(np.arange(1, k // length + 2, dtype=float), length)[:k]
    A = (Q * (lam + 1e-9 * rng.standard_normal(k))) @ Q.T
    A = (A + A.T) / 2
    dA = torch.from_numpy(A.copy()).cuda()
    W = torch.zeros(k, dtype=torch.float64, device="cuda")
    info = torch.ones(1, dtype=torch.int32, device="cuda")
    need = fe.lib.fe_syevd_f64_workspace_bytes(k)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert fe.lib.fe_syevd_f64(dA.data_ptr(), k, k, W.data_ptr(), info.data_ptr(), ws.data_ptr(),
                               need, torch.cuda.current_stream().cuda_stream) == 0
    assert info.item() == 0
    w, Z = W.cpu().numpy(), dA.cpu().numpy().reshape(k, k).T
    nrm = np.abs(A).sum(axis=1).max()
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-12 * nrm
    assert np.abs(A @ Z - Z * w[None, :]).max() <= 1e-12 * nrm
    assert np.abs(Z.T @ Z - np.eye(k)).max() <= 1e-12 * max(k, 10) / 10
